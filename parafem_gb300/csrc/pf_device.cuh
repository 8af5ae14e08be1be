// pf_device.cuh -- device helpers shared by the kernel translation units:
// deterministic reductions and the element routines of the 20-node brick.
#pragma once
#include "pf_internal.h"

#include <cmath>

namespace pf {

#define FULLMASK 0xffffffffu

// ---------------------------------------------------------------------------
// Programmatic dependent launch of an iteration's kernels on small meshes
// (Ctx::dependent): a kernel launched by launch_dependent may start its
// blocks while the one before it drains, which hides the launch.  Such a
// kernel calls pdl_enter() first thing in every thread: it waits until the
// kernel before has completed and its writes are visible.  The kernel before
// calls pdl_exit() in every thread that has done the bulk of its work.  In a
// kernel launched the ordinary way both are no-ops.
// The scatter itself is launched the ordinary way: started early it inherits
// the element kernel's split of the SM, nearly all shared memory, and without
// its L1 it takes twice the time (232 against 113 us on an 80^3 cube).
static __device__ __forceinline__ void pdl_enter() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
static __device__ __forceinline__ void pdl_exit() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
static cudaError_t launch_dependent(bool dependent, cudaStream_t stream, int grid, int block, size_t smem,
                                    void (*kernel)(P...), A... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ---------------------------------------------------------------------------
// reductions
static __device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULLMASK, v, o);
    return v;
}
static __device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(FULLMASK, v, o));
    return v;
}

// A CTA's share of a sum of one value per thread: each warp leaves its
// values in its own `stride` bytes of shared memory (it is done with them),
// the first adds the rows in order.  By all threads of W warps.
template <int W>
static __device__ __forceinline__ void cta_share(unsigned char *rows, int stride, double v, double *out)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncwarp();
    reinterpret_cast<double *>(rows + (size_t)w * stride)[lane] = v;
    __syncthreads();
    if (w > 0) return;
    double s0 = 0.0, s1 = 0.0;   // two chains
#pragma unroll
    for (int j = 0; j < W; j += 2) {
        s0 += reinterpret_cast<const double *>(rows + (size_t)j * stride)[lane];
        s1 += reinterpret_cast<const double *>(rows + (size_t)(j + 1) * stride)[lane];
    }
    s0 = warp_sum(s0 + s1);
    if (lane == 0) *out = s0;
}

// The reductions of the PCG vector kernels (256 threads).  GB300 issues one
// FP64 warp instruction per SM in 16 clocks, so a tree in every warp (eight
// warps x five levels per value) costs more than the sums over a block's
// slots; here one warp per value adds the 256 partial sums from shared
// memory, eight per lane in a fixed order, and runs the one tree.  The sums
// are valid in every thread.
constexpr int kRedThreads = 256;
template <int NV>
static __device__ __forceinline__ void block_sum(double (&v)[NV])
{
    __shared__ double sh[NV][kRedThreads];
    __shared__ double res[NV];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k][t] = v[k];
    __syncthreads();
    if (w < NV) {
        double s = sh[w][lane];
#pragma unroll
        for (int j = 1; j < kRedThreads / 32; ++j) s += sh[w][lane + 32 * j];
        s = warp_sum(s);
        if (lane == 0) res[w] = s;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = res[k];
}

// Maxima of magnitudes, as the bits of their absolute values: those order as
// the values do, so no FP64 compare is needed (a NaN counts as the largest).
static __device__ __forceinline__ long long abs_bits(double x) { return __double_as_longlong(x) & 0x7fffffffffffffffLL; }
static __device__ __forceinline__ void block_max2(long long &a, long long &b)
{
    __shared__ long long sh[2][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = max(a, __shfl_xor_sync(FULLMASK, a, o));
        b = max(b, __shfl_xor_sync(FULLMASK, b, o));
    }
    __syncthreads();
    if (lane == 0) {
        sh[0][w] = a;
        sh[1][w] = b;
    }
    __syncthreads();
    for (int i = 0; i < nw; ++i) {
        a = max(a, sh[0][i]);
        b = max(b, sh[1][i]);
    }
}

// Sums of G block partials (value k at part[k * stride + block]) in a fixed
// order, by one block of 256 threads; valid in every thread.
template <int NV>
static __device__ __forceinline__ void sum_partials(const double *part, size_t stride, int G, double (&v)[NV])
{
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = 0.0;
    for (int i = threadIdx.x; i < G; i += kRedThreads)
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] += __ldcg(part + k * stride + i);
    block_sum<NV>(v);
}

// Maxima of the same two rows of partials (abs_bits held as doubles)
static __device__ __forceinline__ void max_partials2(const double *part, size_t stride, int G, double &ma, double &mb)
{
    long long a = 0, b = 0;
    for (int i = threadIdx.x; i < G; i += blockDim.x) {
        a = max(a, __double_as_longlong(__ldcg(part + i)));
        b = max(b, __double_as_longlong(__ldcg(part + stride + i)));
    }
    block_max2(a, b);
    ma = __longlong_as_double(a);
    mb = __longlong_as_double(b);
}

// True in the block that arrives last of the n that share a counter (in all
// its threads): the others' writes before their arrival are visible to it.
// The counter wraps to zero by itself.  Thread 0 must have made the block's
// writes, or a barrier stand between them and this.
static __device__ __forceinline__ bool last_of(unsigned *count, unsigned n)
{
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicInc(count, n - 1) == n - 1;
    }
    __syncthreads();
    const bool last = s_last != 0;
    if (last) __threadfence();
    return last;
}
static __device__ __forceinline__ bool last_block(unsigned *count) { return last_of(count, gridDim.x); }

// The end of a PCG scatter: the block's share of p.u, and in the last block
// the step length alpha = r.d / p.u.  One thread divides: the vector kernels
// only read the result.
static __device__ __forceinline__ void scatter_tail(double loc, double *part, PcgState *st, unsigned *count)
{
    double v[1] = {loc};
    block_sum<1>(v);
    if (threadIdx.x == 0) part[blockIdx.x] = v[0];
    if (!st || !last_block(count)) return;
    sum_partials<1>(part, 0, gridDim.x, v);
    if (threadIdx.x == 0) st->alpha = st->up / v[0];
}

// Block-uniform read of the stop flag: thread 0 reads it once for the whole
// block, so a block never splits at a barrier when another block of the same
// kernel sets the flag meanwhile.
static __device__ __forceinline__ bool block_stopped(const PcgState *st)
{
    __shared__ int s_stop;
    if (threadIdx.x == 0) s_stop = st ? st->stop : 0;
    __syncthreads();
    const bool v = s_stop != 0;
    __syncthreads();
    return v;
}

// Grid-wide barrier of a cooperative launch (every block resident at once).
// The arrival counter only grows: a block adds one and waits until it
// reaches the next multiple of the block count, which holds while every
// launch that uses the counter has the same block count and completes its
// barriers (the host zeroes it before a run).  Thread 0 releases the
// block's writes before arriving and acquires the others' after the wait.
// The wait is bounded: a block that gives up writes code 3 to *err, sets
// the PCG stop flag (so later launches of the run return at once) and
// returns false; its caller returns, and the blocks still waiting give up
// in turn.  (A two-level form, 16 group counters on separate lines feeding
// a top counter, measured no faster on 600-block grids.)
constexpr long long kGridSpinLimit = 1LL << 22;

static __device__ __forceinline__ bool grid_barrier(unsigned long long *bar, int *err, PcgState *st)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned long long nb = gridDim.x;
        const unsigned long long target = (atomicAdd(bar, 1ULL) / nb + 1) * nb;
        int ok = 0;
        for (long long i = 0; i < kGridSpinLimit; ++i) {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(bar) : "memory");
            if (v >= target) {
                ok = 1;
                break;
            }
            __nanosleep(32);
        }
        if (!ok) {
            atomicExch(err, 3);
            atomicExch(&st->stop, 1);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    const bool ok = s_ok != 0;
    __syncthreads();
    return ok;
}

// SHAPE_DER for one node l of the 20-node brick (new_library.f90:865-896).
static __constant__ int c_xii[20] = {-1, -1, -1, 0, 1, 1, 1, 0, -1, -1, 1, 1, -1, -1, -1, 0, 1, 1, 1, 0};
static __constant__ int c_etai[20] = {-1, -1, -1, -1, -1, -1, -1, -1, 0, 0, 0, 0, 1, 1, 1, 1, 1, 1, 1, 1};
static __constant__ int c_zetai[20] = {-1, 0, 1, 1, 1, 0, -1, -1, -1, 1, 1, -1, -1, 0, 1, 1, 1, 0, -1, -1};

static __device__ __forceinline__ void shape_der20(int l, double xi, double eta, double zeta, double *d)
{
    const double xii = c_xii[l], etai = c_etai[l], zetai = c_zetai[l];
    const double xi0 = xi * xii, eta0 = eta * etai, zeta0 = zeta * zetai;
    const int n = l + 1;
    if (n == 4 || n == 8 || n == 16 || n == 20) {
        d[0] = -.5 * xi * (1. + eta0) * (1. + zeta0);
        d[1] = (.25 * etai) * (1. - xi * xi) * (1. + zeta0);
        d[2] = (.25 * zetai) * (1. - xi * xi) * (1. + eta0);
    } else if (n >= 9 && n <= 12) {
        d[0] = (.25 * xii) * (1. - eta * eta) * (1. + zeta0);
        d[1] = -.5 * eta * (1. + xi0) * (1. + zeta0);
        d[2] = (.25 * zetai) * (1. + xi0) * (1. - eta * eta);
    } else if (n == 2 || n == 6 || n == 14 || n == 18) {
        d[0] = (.25 * xii) * (1. + eta0) * (1. - zeta * zeta);
        d[1] = (.25 * etai) * (1. + xi0) * (1. - zeta * zeta);
        d[2] = -.5 * zeta * (1. + xi0) * (1. + eta0);
    } else {
        d[0] = (.125 * xii) * (1. + eta0) * (1. + zeta0) * (2. * xi0 + eta0 + zeta0 - 1.);
        d[1] = (.125 * etai) * (1. + xi0) * (1. + zeta0) * (xi0 + 2. * eta0 + zeta0 - 1.);
        d[2] = (.125 * zetai) * (1. + xi0) * (1. + eta0) * (xi0 + eta0 + 2. * zeta0 - 1.);
    }
}

// SHAPE_DER for one node l of the 8-node brick (new_library.f90:769-793):
// node signs (xi, eta, zeta) in Smith-Griffiths order, l = 0..7.
static __device__ __forceinline__ void shape_der8(int l, double xi, double eta, double zeta, double *d)
{
    const double sx = (l == 2 || l == 3 || l == 6 || l == 7) ? 1.0 : -1.0;
    const double se = l >= 4 ? 1.0 : -1.0;
    const double sz = (l == 1 || l == 2 || l == 5 || l == 6) ? 1.0 : -1.0;
    const double a = 1.0 + xi * sx, b = 1.0 + eta * se, c = 1.0 + zeta * sz;
    d[0] = 0.125 * sx * b * c;
    d[1] = 0.125 * se * a * c;
    d[2] = 0.125 * sz * a * b;
}

// DEEMAT nst=6 (new_library.f90:1671-1689): the three distinct entries.
static __device__ __forceinline__ void deemat3(double e, double v, double &d11, double &d12, double &d44)
{
    const double v2 = v / (1.0 - v);
    const double vv = (1.0 - 2.0 * v) / (1.0 - v) * 0.5;
    const double den = 2.0 * (1.0 + v) * vv;
    d11 = 1.0 * e / den;
    d12 = v2 * e / den;
    d44 = vv * e / den;
}

// DETERMINANT + INVERT of a 3x3 held column-major (maths.f90:490-633).
static __device__ __forceinline__ double det_invert3(double *m)
{
#define M(a, b) m[((a) - 1) + 3 * ((b) - 1)]
    double det = M(1, 1) * (M(2, 2) * M(3, 3) - M(3, 2) * M(2, 3));
    det = det - M(1, 2) * (M(2, 1) * M(3, 3) - M(3, 1) * M(2, 3));
    det = det + M(1, 3) * (M(2, 1) * M(3, 2) - M(3, 1) * M(2, 2));
    const double j11 = M(2, 2) * M(3, 3) - M(3, 2) * M(2, 3);
    const double j21 = -M(2, 1) * M(3, 3) + M(3, 1) * M(2, 3);
    const double j31 = M(2, 1) * M(3, 2) - M(3, 1) * M(2, 2);
    const double j12 = -M(1, 2) * M(3, 3) + M(3, 2) * M(1, 3);
    const double j22 = M(1, 1) * M(3, 3) - M(3, 1) * M(1, 3);
    const double j32 = -M(1, 1) * M(3, 2) + M(3, 1) * M(1, 2);
    const double j13 = M(1, 2) * M(2, 3) - M(2, 2) * M(1, 3);
    const double j23 = -M(1, 1) * M(2, 3) + M(2, 1) * M(1, 3);
    const double j33 = M(1, 1) * M(2, 2) - M(2, 1) * M(1, 2);
    M(1, 1) = j11 / det; M(1, 2) = j12 / det; M(1, 3) = j13 / det;
    M(2, 1) = j21 / det; M(2, 2) = j22 / det; M(2, 3) = j23 / det;
    M(3, 1) = j31 / det; M(3, 2) = j32 / det; M(3, 3) = j33 / det;
#undef M
    return det;
}


}  // namespace pf
