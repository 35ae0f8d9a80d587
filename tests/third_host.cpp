/* third(x) (dgr_device.cuh) against x / 3 on the host: random bit patterns over the whole
 * range, subnormals, neighbours of powers of two, zeros, infinities.  Returns how many differ
 * in their bits (NaNs count as equal). */
#include <cmath>
#include <cstring>

#include "../dg-rain_b200/csrc/dgr_device.cuh"

static unsigned long long next(unsigned long long &s)
{
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
}

extern "C" long long dgr_t_third(long long n, unsigned long long seed)
{
    long long bad = 0;
    for (long long i = 0; i < n; ++i) {
        unsigned long long u = next(seed);
        if (i % 4 == 1) u = (u & 0x800fffffffffffffull) >> (next(seed) % 53) | (u & (1ull << 63)); /* subnormals */
        if (i % 4 == 2) u = (u & 0xfff0000000000000ull) + (next(seed) % 9) - 4;                     /* powers of two */
        if (i % 64 == 3) u = (u & (1ull << 63)) | (i % 128 == 3 ? 0ull : 0x7ff0000000000000ull);
        double x, a, b;
        memcpy(&x, &u, 8);
        a = dgr::third(x);
        b = x / 3;
        if (std::isnan(b) ? !std::isnan(a) : memcmp(&a, &b, 8) != 0) ++bad;
    }
    return bad;
}
