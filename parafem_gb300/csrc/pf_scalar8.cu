// pf_scalar8.cu -- p123's path: 3-D Laplace (potential flow) with 8-node
// bricks and one freedom per node, solved by the same element-by-element
// Jacobi-PCG (src/programs/5th_ed/p123/p123.f90).
//
// A context set up with pf_setup_scalar8 holds 8-node connectivity, one slot
// per node, and storkc(8,8,e).  The PCG vector kernels are the 20-node path's
// (they work on slots); this file adds:
//   k_form_storkc     kc = sum_gp (kx dx dx' + ky dy dy' + kz dz dz') det w
//                     (p123.f90:70-85), eight threads per element;
//   k_elem8           u_e = kc_e p_e, eight threads per element (thread i
//                     owns row i and reads column j of kc_e as the group's
//                     contiguous 64 bytes), FP64 in ascending column order;
//   k_scatter1        node-centric sum in ascending element order, with
//                     p123's fixed freedoms: u = p * store at a node fixed by
//                     the penalty method (p123.f90:127-131);
//   k_assemble_diag1  the Jacobi diagonal (p123.f90:87-94);
//   k_rows*           the same sums with the element matrices added up by
//                     node once, when storkc is formed: one row of the
//                     assembled matrix per node, and
//   k_row_ring, k_row_product   the product, dot and fixed freedoms in one
//                     pass over the rows.  A node of a brick mesh has 27 neighbours:
//                     270 bytes and 27 FMA per node and product, where the
//                     element products and the scatter move 710 bytes and
//                     take 64 FMA and 8 additions per element.  The element
//                     kernels serve meshes with a node of more than kRowMax
//                     neighbours and contexts without memory for the rows.
#include "pf_device.cuh"
#include "pf_tc.cuh"

#include <algorithm>
#include <vector>

namespace pf {

// Eight threads per element; thread c owns column c of kcx, kcy, kcz.
__global__ void __launch_bounds__(128)
k_form_storkc(int nels, int nip, const double *__restrict__ gp, const double *__restrict__ coord, double kx,
              double ky, double kz, double *__restrict__ kc, double *__restrict__ ediag)
{
    const int c = threadIdx.x & 7;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)nels * 8;
         t += (long long)gridDim.x * blockDim.x) {
        const size_t e = (size_t)(t >> 3);
        const double *co = coord + e * 24;   // coord(8,3)
        double kxx[8], kyy[8], kzz[8];
        for (int r = 0; r < 8; ++r) kxx[r] = kyy[r] = kzz[r] = 0.0;
        for (int g = 0; g < nip; ++g) {
            const double xi = gp[4 * g], eta = gp[4 * g + 1], zeta = gp[4 * g + 2], w = gp[4 * g + 3];
            double der[24];
            for (int l = 0; l < 8; ++l) shape_der8(l, xi, eta, zeta, &der[3 * l]);
            double jac[9];
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) {
                    double s = 0.0;
                    for (int k = 0; k < 8; ++k) s += der[a + 3 * k] * co[k + 8 * b];
                    jac[a + 3 * b] = s;
                }
            const double det = det_invert3(jac);
            double dv[24];
            for (int l = 0; l < 8; ++l)
                for (int a = 0; a < 3; ++a)
                    dv[a + 3 * l] = jac[a] * der[3 * l] + jac[a + 3] * der[3 * l + 1] + jac[a + 6] * der[3 * l + 2];
            for (int r = 0; r < 8; ++r) {
                kxx[r] += dv[3 * r] * dv[3 * c] * det * w;
                kyy[r] += dv[3 * r + 1] * dv[3 * c + 1] * det * w;
                kzz[r] += dv[3 * r + 2] * dv[3 * c + 2] * det * w;
            }
        }
        double *out = kc + e * 64 + 8 * c;
        for (int r = 0; r < 8; ++r) out[r] = kxx[r] * kx + kyy[r] * ky + kzz[r] * kz;
        ediag[e * 8 + c] = out[c];
    }
}

// u_e = kc_e p_e: eight threads per element, thread i owns row i
__global__ void __launch_bounds__(256)
k_elem8(int nels, const double *__restrict__ kc, const int *__restrict__ conn, const double *__restrict__ p,
        double *__restrict__ ut, const PcgState *__restrict__ st)
{
    pdl_enter();
    if (st && st->stop) return;
    const int i = threadIdx.x & 7;
    const unsigned gmask = 0xFFu << (threadIdx.x & 24);   // the 8 lanes of this element
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)nels * 8;
         t += (long long)gridDim.x * blockDim.x) {
        const size_t e = (size_t)(t >> 3);
        const double pi = p[conn[e * 8 + i]];
        const double *k = kc + e * 64 + i;
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc = fma(k[8 * j], __shfl_sync(gmask, pi, (threadIdx.x & 24) + j), acc);
        ut[e * 8 + i] = acc;
    }
}

// Node-centric scatter (one freedom per node).  list[] holds e*8+a.
//   MODE 0: out = u, partial p.u          (pf = p)
//   MODE 1: out = f - u, partial out.out  (pf = f)
// A fixed node (fstore != 0) takes u = p * store (p123.f90:127-131);
// a restrained node gets 0.
template <int MODE>
__global__ void __launch_bounds__(256)
k_scatter1(int nn, const int *__restrict__ ptr, const int *__restrict__ list, const double *__restrict__ ut,
           const uint8_t *__restrict__ fm, const double *__restrict__ fstore, const double *__restrict__ xin,
           const double *__restrict__ pf, double *__restrict__ out, double *__restrict__ part,
           PcgState *st, unsigned *__restrict__ count)
{
    if (st && st->stop) return;
    double loc = 0.0;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += gridDim.x * blockDim.x) {
        double a = 0.0;
        for (int k = ptr[n]; k < ptr[n + 1]; ++k) a += ut[list[k]];
        const bool fr = fm[n] & 1;
        const double fs = fstore[n];
        if (fs != 0.0) a = xin[n] * fs;
        if (MODE == 0) {
            const double uv = fr ? a : 0.0;
            out[n] = uv;
            loc = fma(pf[n], uv, loc);
        } else {
            const double rv = fr ? pf[n] - a : 0.0;
            out[n] = rv;
            loc = fma(rv, rv, loc);
        }
    }
    pdl_exit();
    scatter_tail(loc, part, MODE == 0 ? st : nullptr, count);
}

// ---------------------------------------------------------------------------
// Assembled rows, in slices of 32 consecutive nodes: entry k of the rows of
// slice s lies at off[s] + 32 k + lane, columns ascending.  Column numbers are
// 16-bit offsets from the least column of (slice, k) where every one fits
// (neighbouring nodes have neighbouring columns), 32-bit numbers otherwise.
// Short rows are padded with 0 at a column of their own: at another node's,
// 0 x Inf or 0 x NaN would carry that node's value into a row that is not its
// neighbour.  Where no column of its own lies within 16 bits (the last layer
// of a mesh with more than 65,535 nodes per layer) the row is padded with
// -0.0, which no sum that starts from 0 is, and the products step over it
// (SKIP; in all meshes that test would cost 1.5 % of an iteration).
constexpr int kRowMax = 64;   // entries of a row (a structured brick mesh has 27)

// the ascending distinct columns of node n: their number, -1 when too many
__device__ int row_columns(int n, const int *__restrict__ ptr, const int *__restrict__ list,
                           const int *__restrict__ conn, int *cols)
{
    int cnt = 0;
    for (int q = ptr[n]; q < ptr[n + 1]; ++q) {
        const int *ce = conn + (size_t)(list[q] >> 3) * 8;
        for (int j = 0; j < 8; ++j) {
            const int c = ce[j];
            int m = cnt;
            while (m > 0 && cols[m - 1] > c) --m;
            if (m > 0 && cols[m - 1] == c) continue;
            if (cnt == kRowMax) return -1;
            for (int i = cnt; i > m; --i) cols[i] = cols[i - 1];
            cols[m] = c;
            ++cnt;
        }
    }
    return cnt;
}

__global__ void __launch_bounds__(128)
k_rows_width(int nn, const int *__restrict__ ptr, const int *__restrict__ list, const int *__restrict__ conn,
             int *__restrict__ width, int *__restrict__ bad)
{
    const int nslice = (nn + 31) / 32, lane = threadIdx.x & 31;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslice; s += (gridDim.x * blockDim.x) >> 5) {
        int cols[kRowMax];
        const int n = 32 * s + lane;
        const int cnt = n < nn ? row_columns(n, ptr, list, conn, cols) : 0;
        if (cnt < 0) atomicOr(bad, 1);
        const int w = __reduce_max_sync(FULLMASK, cnt);
        if (lane == 0) width[s] = w;
    }
}

template <bool SKIP>
__device__ __forceinline__ double row_step(double k, double x, double a)
{
    return SKIP && __double_as_longlong(k) == (long long)0x8000000000000000ULL ? a : fma(k, x, a);
}

// Values summed in ascending element order; *bad, bit 0: a 16-bit offset
// overflows, bit 1: rows padded with -0.0.
template <typename IT>
__global__ void __launch_bounds__(128)
k_rows_fill(int nn, const int *__restrict__ ptr, const int *__restrict__ list, const int *__restrict__ conn,
            const double *__restrict__ kc, const long long *__restrict__ off, double *__restrict__ val,
            IT *__restrict__ idx, int *__restrict__ base, int *__restrict__ bad)
{
    const int nslice = (nn + 31) / 32, lane = threadIdx.x & 31;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslice; s += (gridDim.x * blockDim.x) >> 5) {
        int cols[kRowMax];
        double v[kRowMax];
        const int n = 32 * s + lane;
        int cnt = 0;
        if (n < nn) {
            cnt = row_columns(n, ptr, list, conn, cols);
            for (int k = 0; k < cnt; ++k) v[k] = 0.0;
            for (int q = ptr[n]; q < ptr[n + 1]; ++q) {
                const size_t e = (size_t)(list[q] >> 3);
                const int a = list[q] & 7;
                for (int j = 0; j < 8; ++j) {
                    const int c = conn[e * 8 + j];
                    int k = 0;
                    while (cols[k] != c) ++k;
                    v[k] += kc[e * 64 + a + 8 * j];
                }
            }
        }
        const long long o = off[s];
        const int w = (int)((off[s + 1] - o) >> 5);
        for (int k = 0; k < w; ++k) {
            const int first = __reduce_min_sync(FULLMASK, k < cnt ? cols[k] : 0x7fffffff);
            int c = k < cnt ? cols[k] : first;   // (a row without columns is no freedom's)
            if (k >= cnt && cnt > 0)             // its least column from `first` on, or its last
                for (int m = cnt - 1; m >= 0 && (m == cnt - 1 || cols[m] >= first); --m) c = cols[m];
            int least = __reduce_min_sync(FULLMASK, c);
            double pad = 0.0;
            if (sizeof(IT) == 2 && __any_sync(FULLMASK, c - least > 0xffff)) {
                least = first;
                if (k >= cnt) {
                    c = first;
                    pad = -0.0;
                }
                atomicOr(bad, c - least > 0xffff ? 1 : 2);
            }
            val[o + 32 * k + lane] = k < cnt ? v[k] : pad;
            idx[o + 32 * k + lane] = (IT)(sizeof(IT) == 2 ? c - least : c);
            if (lane == 0) base[(o >> 5) + k] = least;
        }
    }
}

// u = K x over the assembled rows, as k_elem8 and k_scatter1 form it:
//   MODE 0: out = u, partial pf.u and alpha in a PCG run;  MODE 1: out = f - u, partial out.out
// For MODE 0 where k_row_ring does not take the rows.  Bound by the FP64 pipe
// (30 operations per node, two per SM and clock: 56 us at 100^3) and by HBM
// (294 B per node, 44 us), one after the other: 92 us at 100^3, where k_elem8
// and k_scatter1 take 180.  KEEP: the rows are read the ordinary way, so that
// those of a mesh that fits stay in L2 from one product to the next; else they
// leave L2 first (100^3: 98 us kept, 90 us not).
constexpr size_t kRowKeepBytes = 64u << 20;
template <int MODE, typename IT, bool KEEP, bool SKIP>
__global__ void __launch_bounds__(256)
k_row_product(int nn, const long long *__restrict__ off, const double *__restrict__ val, const IT *__restrict__ idx,
              const int *__restrict__ base, const uint8_t *__restrict__ fm, const double *__restrict__ fstore,
              const double *__restrict__ xin, const double *__restrict__ pf, double *__restrict__ out,
              double *__restrict__ part, PcgState *st, unsigned *__restrict__ count)
{
    pdl_enter();
    if (st && st->stop) return;
    double loc = 0.0;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += gridDim.x * blockDim.x) {
        const int s = n >> 5, lane = n & 31;
        const long long o = off[s];
        const int w = (int)((off[s + 1] - o) >> 5);
        const double *v = val + o + lane;
        const IT *ix = idx + o + lane;
        const int *b = base + (o >> 5);
        double a = 0.0;
#pragma unroll 9
        for (int k = 0; k < w; ++k) {
            const int i = (int)(KEEP ? __ldg(ix + 32 * k) : __ldcs(ix + 32 * k));
            const int c = sizeof(IT) == 2 ? __ldg(b + k) + i : i;
            a = row_step<SKIP>(KEEP ? __ldg(v + 32 * k) : __ldcs(v + 32 * k), __ldg(xin + c), a);
        }
        const bool fr = fm[n] & 1;
        const double fs = fstore[n];
        if (abs_bits(fs)) a = xin[n] * fs;   // an integer test
        if (MODE == 0) {
            const double uv = fr ? a : 0.0;
            out[n] = uv;
            loc = fma(pf[n], uv, loc);
        } else {
            const double rv = fr ? pf[n] - a : 0.0;
            out[n] = rv;
            loc = fma(rv, rv, loc);
        }
    }
    pdl_exit();
    scatter_tail(loc, part, MODE == 0 ? st : nullptr, count);
}

// k_row_product<0> with the rows streamed through shared memory: one
// persistent CTA of 20 warps per SM, one warp per slice of 32 rows; each warp
// has the next slice's values and columns copied (cp.async.bulk) while the
// other warps multiply, so that the memory and the FP64 pipe are busy
// together.  The sums are k_row_product's, in its order.  Every wait on an
// mbarrier is bounded, as in k_elem_sym32.  Bound by the FP64 pipe (50 us at
// 100^3): 70 us, where k_row_product takes 92; 150^3 198 against 259, 32^3
// 12.2 against 16.4 (fewer blocks to sum over), 50^3 to 64^3 alike.  8, 12, 16
// and 24 warps: 92, 75, 71, 71 us at 100^3.
// Rule: slices of at most 28 columns (27 in a mesh of bricks) with 16-bit
// column offsets.
constexpr int kRingWarps = 20, kRingWidth = 28;                  // widest slice that a stage holds
constexpr int kRingIdx = kRingWidth * 32 * 8, kRingStage = kRingWidth * 32 * 10;
constexpr int kRingSmem = kRingWarps * (kRingStage + 8);
static_assert(kRingSmem + 64 <= 227 * 1024, "shared memory per CTA");
template <bool SKIP>
__global__ void __launch_bounds__(kRingWarps * 32, 1)
k_row_ring(int nn, const long long *__restrict__ off, const double *__restrict__ val, const uint16_t *__restrict__ idx,
           const int *__restrict__ base, const uint8_t *__restrict__ fm, const double *__restrict__ fstore,
           const double *__restrict__ xin, double *__restrict__ out, double *__restrict__ part, PcgState *st,
           unsigned *__restrict__ count, int keep, int *__restrict__ err)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned char *stage = smem + (size_t)w * kRingStage;
    const double *sv = reinterpret_cast<const double *>(stage) + lane;
    const uint16_t *si = reinterpret_cast<const uint16_t *>(stage + kRingIdx) + lane;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + (size_t)kRingWarps * kRingStage) + w;
    // this CTA's contiguous range of slices, warps interleaved inside it
    const int nslice = (nn + 31) / 32, per_cta = (nslice + gridDim.x - 1) / gridDim.x;
    const int s1 = min(nslice, (int)(blockIdx.x + 1) * per_cta);
    int s = blockIdx.x * per_cta + w;
    const uint64_t pol = tc::l2_evict_first_policy();
    auto issue = [&](long long o, int n) {   // n columns from entry o on (lane 0)
        tc::mbar_expect_tx(bar, n * 320);
        if (keep) {
            tc::bulk_g2s(stage, val + o, n * 256, bar);
            tc::bulk_g2s(stage + kRingIdx, idx + o, n * 64, bar);
        } else {
            tc::bulk_g2s_hint(stage, val + o, n * 256, bar, pol);
            tc::bulk_g2s_hint(stage + kRingIdx, idx + o, n * 64, bar, pol);
        }
    };
    long long o = 0;
    int n = 0;
    if (s < s1) {   // the rows are no kernel's of this iteration: before the wait for the one before
        o = off[s];
        n = (int)((off[s + 1] - o) >> 5);
        if (lane == 0) {
            tc::mbar_init(bar, 1);
            tc::mbar_fence_init();
            issue(o, n);
        }
    }
    __syncwarp();
    pdl_enter();
    const bool stopped = st && st->stop;
    double loc = 0.0;
    bool ok = true;
    for (uint32_t parity = 0; s < s1; s += kRingWarps, parity ^= 1) {
        const int b = lane < n ? __ldg(base + (o >> 5) + lane) : 0;
        const int row = 32 * s + lane;
        const bool in = row < nn;
        const int m = in ? fm[row] : 0;
        const double fs = in ? fstore[row] : 0.0, p = in ? xin[row] : 0.0;
        ok = __all_sync(FULLMASK, tc::mbar_wait(bar, parity));
        if (!ok || stopped) break;
        double a = 0.0;
#pragma unroll 9
        for (int k = 0; k < n; ++k) a = row_step<SKIP>(sv[32 * k], __ldg(xin + __shfl_sync(FULLMASK, b, k) + si[32 * k]), a);
        __syncwarp();   // every lane is done with the stage
        if (s + kRingWarps < s1) {
            o = off[s + kRingWarps];
            n = (int)((off[s + kRingWarps + 1] - o) >> 5);
            if (lane == 0) {
                tc::fence_proxy_async();
                issue(o, n);
            }
        }
        if (in) {
            if (abs_bits(fs)) a = p * fs;   // an integer test
            const double uv = m & 1 ? a : 0.0;
            out[row] = uv;
            loc = fma(p, uv, loc);
        }
    }
    if (stopped) return;
    if (!ok && lane == 0) {
        atomicExch(err, 2);
        tc::mbar_wait(bar, 0);   // the one copy in flight, once more (bounded)
        tc::mbar_wait(bar, 1);
    }
    pdl_exit();
    cta_share<kRingWarps>(smem, kRingStage, loc, part + blockIdx.x);
    if (!st || w > 0) return;
    int last = 0;
    if (lane == 0) {
        __threadfence();
        last = atomicInc(count, gridDim.x - 1) == gridDim.x - 1;
    }
    if (!__shfl_sync(FULLMASK, last, 0)) return;
    __threadfence();
    double v = 0.0;
    for (int i = lane; i < (int)gridDim.x; i += 32) v += __ldcg(part + i);
    v = warp_sum(v);
    if (lane == 0) st->alpha = st->up / v;
}

__global__ void k_assemble_diag1(int nn, const int *__restrict__ ptr, const int *__restrict__ list,
                                 const double *__restrict__ ed, const uint8_t *__restrict__ fm,
                                 double *__restrict__ diag, double *__restrict__ dinv, double *__restrict__ fstore)
{
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nn; n += gridDim.x * blockDim.x) {
        double a = 0.0;
        for (int k = ptr[n]; k < ptr[n + 1]; ++k) a += ed[list[k]];
        const bool fr = fm[n] & 1;
        diag[n] = fr ? a : 0.0;
        dinv[n] = fr ? 1.0 / a : 0.0;
        fstore[n] = 0.0;
    }
}

// fixed freedoms (p123.f90:104-110): diag += penalty, store = diag
__global__ void k_set_fixed(int nfix, const int *__restrict__ slots, double penalty, double *__restrict__ diag,
                            double *__restrict__ dinv, double *__restrict__ fstore)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nfix; i += gridDim.x * blockDim.x) {
        const int s = slots[i];
        const double d = diag[s] + penalty;
        diag[s] = d;
        dinv[s] = 1.0 / d;
        fstore[s] = d;
    }
}

static int launched8(Ctx &c, const char *name)
{
    c.launches++;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s: launch failed: %s", name, cudaGetErrorString(e));
        return 1;
    }
    return 0;
}

static int grid8(const Ctx &c, long long work, int per_block, int max_per_sm)
{
    long long g = (work + per_block - 1) / per_block;
    if (g > (long long)c.nsm * max_per_sm) g = (long long)c.nsm * max_per_sm;
    return (int)(g < 1 ? 1 : g);
}

int launch_form_storkc(Ctx &c, int nip, double kx, double ky, double kz)
{
    double *gp = nullptr;
    if (cudaMallocAsync(&gp, sizeof(double) * 4 * 27, c.stream) != cudaSuccess) {
        set_error("form_storkc: cannot allocate the Gauss table");
        return 1;
    }
    if (launch_sample(c.stream, nip, false, gp)) return 1;
    c.launches++;
    k_form_storkc<<<grid8(c, (long long)c.nels * 8, 128, 16), 128, 0, c.stream>>>(c.nels, nip, gp, c.coord, kx, ky,
                                                                                   kz, c.km64, c.ediag);
    if (launched8(c, "k_form_storkc")) return 1;
    cudaFreeAsync(gp, c.stream);
    return 0;
}

void rows_release(Ctx &c)
{
    void *p[] = {c.row_off, c.row_val, c.row_idx, c.row_base};
    for (void *q : p)
        if (q) cudaFree(q);
    c.row_off = nullptr;
    c.row_val = nullptr;
    c.row_idx = nullptr;
    c.row_base = nullptr;
    c.row_wide = c.row_keep = c.row_skip = c.row_ring = false;
}

// A kernel of the assembly was launched: 0, 1 (failed), or -1 where it found
// no memory (its rows are assembled in local memory)
static int rows_launched(Ctx &c, const char *name)
{
    const cudaError_t e = cudaPeekAtLastError();
    if (e == cudaErrorMemoryAllocation || e == cudaErrorLaunchOutOfResources) {
        cudaGetLastError();
        return -1;
    }
    return launched8(c, name);
}

// The result of rows_assemble, -1 where the memory does not suffice
static int rows_build(Ctx &c)
{
    const int nslice = (c.nn + 31) / 32, grid = grid8(c, c.nn, 128, 16);
    int *d_width = nullptr, bad = 0;
    std::vector<int> width(nslice);
    std::vector<long long> off(nslice + 1, 0);
    if (cudaMalloc((void **)&d_width, (size_t)nslice * sizeof(int)) != cudaSuccess) return -1;
    cudaMemsetAsync(c.kerr + 1, 0, sizeof(int), c.stream);
    k_rows_width<<<grid, 128, 0, c.stream>>>(c.nn, c.node_ptr, c.node_list, c.conn, d_width, c.kerr + 1);
    const int err = rows_launched(c, "k_rows_width");
    cudaMemcpyAsync(width.data(), d_width, (size_t)nslice * sizeof(int), cudaMemcpyDeviceToHost, c.stream);
    cudaMemcpyAsync(&bad, c.kerr + 1, sizeof(int), cudaMemcpyDeviceToHost, c.stream);
    const cudaError_t e = cudaStreamSynchronize(c.stream);
    cudaFree(d_width);
    if (err) return err;
    if (e != cudaSuccess) {
        set_error("k_rows_width: %s", cudaGetErrorString(e));
        return 1;
    }
    if (bad) return 0;
    for (int s = 0; s < nslice; ++s) off[s + 1] = off[s] + 32LL * width[s];
    const auto w = std::minmax_element(width.begin(), width.end());
    const size_t total = (size_t)off[nslice];
    if (total == 0) return 0;
    if (cudaMalloc((void **)&c.row_off, (size_t)(nslice + 1) * sizeof(long long)) != cudaSuccess ||
        cudaMalloc((void **)&c.row_val, total * sizeof(double)) != cudaSuccess ||
        cudaMalloc((void **)&c.row_base, total / 32 * sizeof(int)) != cudaSuccess)
        return -1;
    cudaMemcpyAsync(c.row_off, off.data(), off.size() * sizeof(long long), cudaMemcpyHostToDevice, c.stream);
    for (int bytes = 2; bytes <= 4; bytes += 2) {   // 16-bit columns first
        if (cudaMalloc(&c.row_idx, total * bytes) != cudaSuccess) return -1;
        cudaMemsetAsync(c.kerr + 1, 0, sizeof(int), c.stream);
        if (bytes == 2)
            k_rows_fill<uint16_t><<<grid, 128, 0, c.stream>>>(c.nn, c.node_ptr, c.node_list, c.conn, c.km64, c.row_off,
                                                              c.row_val, (uint16_t *)c.row_idx, c.row_base, c.kerr + 1);
        else
            k_rows_fill<int><<<grid, 128, 0, c.stream>>>(c.nn, c.node_ptr, c.node_list, c.conn, c.km64, c.row_off,
                                                         c.row_val, (int *)c.row_idx, c.row_base, c.kerr + 1);
        const int ef = rows_launched(c, "k_rows_fill");
        if (ef) return ef;
        cudaMemcpyAsync(&bad, c.kerr + 1, sizeof(int), cudaMemcpyDeviceToHost, c.stream);
        const cudaError_t es = cudaStreamSynchronize(c.stream);
        if (es != cudaSuccess) {
            set_error("k_rows_fill: %s", cudaGetErrorString(es));
            return 1;
        }
        if (!(bad & 1)) {
            c.row_wide = bytes == 4;
            c.row_keep = total * (8 + bytes) <= kRowKeepBytes;
            c.row_skip = bad != 0;
            c.row_ring = bytes == 2 && *w.first > 0 && *w.second <= kRingWidth;
            break;
        }
        cudaFree(c.row_idx);
        c.row_idx = nullptr;
    }
    return 0;
}

// The assembled rows of the context's storkc; none (and success) where a row
// is too long or the memory does not suffice, none either after an error:
// rows that are there are whole.
int rows_assemble(Ctx &c)
{
    rows_release(c);
    const int rc = rows_build(c);
    if (rc == 0) return 0;
    cudaGetLastError();
    rows_release(c);
    return rc > 0;
}

static int launch_row_product(Ctx &c, int mode, const double *xin, const double *pf, double *out, PcgState *st)
{
    if (mode == 0 && c.row_ring) {
        if (!c.row_attr) {   // by the first product, outside any stream capture
            cudaError_t e = cudaFuncSetAttribute(k_row_ring<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRingSmem);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k_row_ring<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRingSmem);
            if (e != cudaSuccess) {
                set_error("k_row_ring: cannot reserve %d bytes of shared memory: %s", kRingSmem, cudaGetErrorString(e));
                return 1;
            }
            c.row_attr = true;
        }
        const int grid = c.Gs < c.nsm ? c.Gs : c.nsm;   // c.part_s holds c.Gs shares
        launch_dependent(c.dependent && st, c.stream, grid, kRingWarps * 32, kRingSmem,
                         c.row_skip ? k_row_ring<true> : k_row_ring<false>, c.nn, c.row_off, c.row_val, (const uint16_t *)c.row_idx,
                         c.row_base, c.freemask, c.fstore, xin, out, c.part_s, st, c.count,
                         c.row_keep ? 1 : 0, c.kerr);
        return launched8(c, "k_row_ring");
    }
    auto go = [&](auto *idx, auto kernel0, auto kernel1) {
        launch_dependent(c.dependent && st, c.stream, c.Gs, 256, 0, mode ? kernel1 : kernel0, c.nn, c.row_off, c.row_val,
                         idx, c.row_base, c.freemask, c.fstore, xin, pf, out, c.part_s, st, c.count);
    };
    const int *wide = (const int *)c.row_idx;
    const uint16_t *narrow = (const uint16_t *)c.row_idx;
    if (c.row_wide) go(wide, k_row_product<0, int, false, false>, k_row_product<1, int, false, false>);
    else if (c.row_skip) go(narrow, k_row_product<0, uint16_t, false, true>, k_row_product<1, uint16_t, false, true>);
    else if (c.row_keep) go(narrow, k_row_product<0, uint16_t, true, false>, k_row_product<1, uint16_t, true, false>);
    else go(narrow, k_row_product<0, uint16_t, false, false>, k_row_product<1, uint16_t, false, false>);
    return launched8(c, "k_row_product");
}

// The element products; with assembled rows nothing: launch_scatter1 forms
// the whole product.
int launch_elem8(Ctx &c, const double *p, const PcgState *st)
{
    if (c.row_idx) return 0;
    launch_dependent(c.dependent && st, c.stream, grid8(c, (long long)c.nels * 8, 256, 8), 256, 0, k_elem8, c.nels, c.km64, c.conn, p,
                     (double *)c.utemp, st);
    return launched8(c, "k_elem8");
}

int launch_scatter1(Ctx &c, int mode, const double *xin, const double *pf, double *out, PcgState *st)
{
    if (c.row_idx) return launch_row_product(c, mode, xin, pf, out, st);
    if (mode == 0)
        k_scatter1<0><<<c.Gs, 256, 0, c.stream>>>(c.nn, c.node_ptr, c.node_list, (const double *)c.utemp, c.freemask,
                                                  c.fstore, xin, pf, out, c.part_s, st, c.count);
    else
        k_scatter1<1><<<c.Gs, 256, 0, c.stream>>>(c.nn, c.node_ptr, c.node_list, (const double *)c.utemp, c.freemask,
                                                  c.fstore, xin, pf, out, c.part_s, st, c.count);
    return launched8(c, "k_scatter1");
}

int launch_assemble_diag1(Ctx &c)
{
    k_assemble_diag1<<<grid8(c, c.nn, 256, 8), 256, 0, c.stream>>>(c.nn, c.node_ptr, c.node_list, c.ediag,
                                                                    c.freemask, c.diag, c.dinv, c.fstore);
    return launched8(c, "k_assemble_diag1");
}

int launch_set_fixed(Ctx &c, int nfix, const int *slots_dev, double penalty)
{
    k_set_fixed<<<grid8(c, nfix, 256, 4), 256, 0, c.stream>>>(nfix, slots_dev, penalty, c.diag, c.dinv, c.fstore);
    return launched8(c, "k_set_fixed");
}

}  // namespace pf
