/* The checked build's limiter (dgr_kernels.cuh with DGR_CHECKED) on the host: one element whose
 * node bounds come from the element means (k_fold_limit), with an index out of range among those
 * it gathers.  Returns the recorded word, (kernel << 32 | item), and in *touched whether the
 * element's state or status was written. */
#include <cmath>
#include <cstddef>
#include <cstring>
#include <type_traits>
#include <vector>

/* what the header names of CUDA's device language; none of it runs here but atomicMin, __ldcg */
struct Dim {
    unsigned x;
};
static Dim threadIdx, blockIdx, blockDim, gridDim;
template <class T>
static T atomicMin(T *p, T v)
{
    const T o = *p;
    if (v < o) *p = v;
    return o;
}
template <class T>
static T __ldcg(const T *p) { return *p; }
unsigned long long atomicMax(unsigned long long *, unsigned long long);
unsigned atomicAdd(unsigned *, unsigned);
unsigned atomicExch(unsigned *, unsigned);
double __shfl_xor_sync(unsigned, double, int);
int __shfl_sync(unsigned, int, int);
bool __all_sync(unsigned, bool);
void __syncthreads();
int __syncthreads_and(int);
void __threadfence();
void __nanosleep(unsigned);
size_t __cvta_generic_to_global(const void *);
size_t __cvta_generic_to_shared(const void *);
long long __double_as_longlong(double);
double __longlong_as_double(long long);
template <class A, class B>
static std::common_type_t<A, B> min(A a, B b) { return a < b ? a : b; }
template <class A, class B>
static std::common_type_t<A, B> max(A a, B b) { return a > b ? a : b; }
using std::isnan;

#define DGR_CHECKED
#include "../dg-rain_b200/csrc/dgr_scheme.cuh"
#undef DGR_HD
#include "../dg-rain_b200/csrc/dgr_kernels.cuh"

using namespace dgr;

/* element 1 of 40 at nodes 0, 1, 2 with `many` elements around each node; where: 0 nothing wrong,
 * 1 the element's node, 2 the bounds of a node's list, 3 an early entry of a list, 4 one past the
 * entries prepared ahead, 5 an empty list */
extern "C" unsigned long long dgr_t_bad_index(int where, int *touched)
{
    const int ne = 40, nn = 4, many = 9, el = 1;
    std::vector<int> el2v(3 * ne, 0), ptr(nn + 1), n2e(nn * many);
    for (int n = 0; n <= nn; ++n) ptr[n] = n * many;
    for (int j = 0; j < nn * many; ++j) n2e[j] = j;
    for (int k = 0; k < 3; ++k) el2v[k * ne + el] = k;
    std::vector<double> zn(nn, 5.0), avg(3 * ne, 0.25), S(9 * ne, 0.25);
    std::vector<int> in(ne, 1), out(ne, -7);
    DevClock clk;
    memset(&clk, 0, sizeof clk);
    clk.err = ~0ull;
    if (where == 1) el2v[2 * ne + el] = nn;
    if (where == 2) ptr[2] = -1;
    if (where == 3) n2e[many + 1] = ne;
    if (where == 4) n2e[many + 8] = -1;
    if (where == 5) ptr[2] = ptr[3];
    unsigned long long bad = ~0ull;
    MeshDev m;
    memset(&m, 0, sizeof m);
    m.ne = m.ldE = ne;
    m.nn = m.ldN = nn;
    m.el2v = el2v.data();
    m.n2e_ptr = ptr.data();
    m.n2e = n2e.data();
    m.zn = zn.data();
    m.bad_index = &bad;
    const std::vector<double> was = S;
    limit_item<true, true, true, true, true>(m, S.data(), avg.data(), in.data(), out.data(), &clk, 1e-3, 1e-2, 1, nullptr,
                                             nullptr, el);
    *touched = S != was || out[el] != -7;
    return bad;
}

/* the three edges of element 1 of 4, edge `at` (or none, -1) one past the last of 9 */
extern "C" unsigned long long dgr_t_bad_edge(int at, int *ok)
{
    const int ne = 4, nf = 9, el = 1;
    std::vector<int> ee(3 * ne);
    for (int j = 0; j < 3 * ne; ++j) ee[j] = 2 * (j % nf) + j % 2;
    if (at >= 0) ee[at * ne + el] = 2 * nf + 1;
    unsigned long long bad = ~0ull;
    MeshDev m;
    memset(&m, 0, sizeof m);
    m.ne = m.ldE = ne;
    m.nf = nf;
    m.elem_edge = ee.data();
    m.bad_index = &bad;
    *ok = element_edges_ok(m, el);
    return bad;
}
