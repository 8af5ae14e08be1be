// pf_resident.cu -- whole PCG runs of small meshes in one cooperative launch.
//
// On a small mesh an iteration of four kernels is launch latency: 22 us on
// 10^3 elements, of which the chip works perhaps three.  Here one CTA per SM
// (of half the SMs on the smallest meshes) stays for the whole run.  A CTA
// owns a range of elements and a range of slots; its elements' records stay in shared memory when they fit (14 FP64,
// 28 FP32 or 48 FP16 records per SM: 12.8^3, 16^3, 19^3 elements on 152 SMs)
// and stream through it otherwise.  An iteration (p121.f90:90-104 with
// DOT_PRODUCT_P, maths.f90:168-215, and checon_par, maths.f90:1052-1062) is
// two phases with one grid-wide exchange after each:
//   elements  u_e = K_e p_e with p = d + beta p_old formed in the gather, so
//             that p needs no phase of its own; results to utemp; share of
//             p.u as the sum of p_e.u_e
//   slots     u = sum over a node's elements; the owner keeps p; x, r, d;
//             shares of r.d and r.r (or checon_par's maxima)
// (With p.u formed from the summed u, a third exchange stands between u and
// x: 13.5 us per iteration on 10^3 elements.)
// An exchange is one counter that every CTA adds to (red.release) and one
// thread of every CTA polls (ld.acquire): 1.2 us over 152 CTAs, where tagged
// words that all CTAs poll took 2.1 us and words pushed into a mailbox per
// CTA 3.8.  The CTAs' shares of a sum lie in memory beside it; every CTA adds
// them in the same fixed order, so all decide alike and runs are bitwise
// reproducible.  Every wait is bounded: one that runs out records code 3 and
// stops the run.
#include "pf_fix.cuh"
#include "pf_sym.cuh"

namespace pf {

namespace {

constexpr int kResThreads = 512;
constexpr int kMaxBlocks = kShareBlocks;   // shares a warp adds: eight per lane

struct ResArgs {
    int nels, ns, niters, per_slots;
    const unsigned char *rec;
    size_t stride;               // bytes from element to element: 0 for one matrix (FP64)
    const int *conn;
    void *ut;
    const int *ptr, *list;
    const uint8_t *fm;
    double *x, *r, *d, *p;
    const double *dinv;
    PcgState *st;
    unsigned long long *count;   // arrivals, zero at the launch
    double *part;                // [4][kMaxBlocks] shares: p.u, r.d, r.r or max |x|, max |dx|
    int *kerr;
};

// per precision: warps that form products, ring stages per warp, bytes of a
// stage and of the warp's p words
template <int PREC> struct Shape;
template <> struct Shape<64> { static constexpr int W = 14, S = 1, stage = 3 * fx::kChunk0, pbytes = 960, rec = fx::kRecBytes; };
template <> struct Shape<32> { static constexpr int W = 14, S = 2, stage = sym::kBytes32, pbytes = 480, rec = sym::kBytes32; };
template <> struct Shape<16> { static constexpr int W = 16, S = 3, stage = sym::kBytes16, pbytes = 480, rec = sym::kBytes16; };
// the p words double as the block sums' scratch (two doubles per thread)
template <int PREC> constexpr int kScratch = Shape<PREC>::W * Shape<PREC>::pbytes > kResThreads * 16
                                                 ? Shape<PREC>::W * Shape<PREC>::pbytes : kResThreads * 16;
template <int PREC> constexpr size_t kResSmem =
    (size_t)Shape<PREC>::W * Shape<PREC>::S * Shape<PREC>::stage + kScratch<PREC> + Shape<PREC>::W * 3 * 8;

// One thread: its block's writes are out (with those of the threads it has
// met at a barrier), and every block's are visible on return; false when the
// wait ran out.
__device__ __forceinline__ bool exchange(unsigned long long *count, unsigned long long target,
                                         long long polls = kGridSpinLimit)
{
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(count), "l"(1ULL) : "memory");
    for (long long i = 0; i < polls; ++i) {
        unsigned long long v;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(count) : "memory");
        if (v >= target) return true;
    }
    return false;
}

// ||r|| <= tol ||f|| as a bound for r.r: a negative tolerance is never met
__device__ __forceinline__ double stop_square(double tol, double root_ff)
{
    const double b = tol * root_ff;
    return tol >= 0.0 ? b * b : -1.0;
}

// One warp: the blocks' shares added (or their greatest bits), in every lane
__device__ __forceinline__ double add_shares(const double *p, int nblk, int lane)
{
    double v[kMaxBlocks / 32];
#pragma unroll
    for (int j = 0; j < kMaxBlocks / 32; ++j) v[j] = lane + 32 * j < nblk ? __ldcg(p + lane + 32 * j) : 0.0;
    double s = v[0];
#pragma unroll
    for (int j = 1; j < kMaxBlocks / 32; ++j)
        if (32 * j < nblk) s += v[j];
    return warp_sum(s);
}
__device__ __forceinline__ long long max_shares(const double *p, int nblk, int lane)
{
    long long m = 0;
#pragma unroll
    for (int j = 0; j < kMaxBlocks / 32; ++j)
        if (lane + 32 * j < nblk) m = max(m, __double_as_longlong(__ldcg(p + lane + 32 * j)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(FULLMASK, m, o));
    return m;
}

}  // namespace

// One exchange that nothing completes, as pf_check_wait_timeout runs it
__global__ void k_exchange_probe(unsigned long long *count, long long polls, int *kerr)
{
    if (threadIdx.x == 0 && !exchange(count, ~0ULL, polls)) atomicExch(kerr, 3);
}

template <int PREC, bool CHECON, int NSL>
__global__ void __launch_bounds__(kResThreads, 1) k_pcg_resident(ResArgs a)
{
    using Sh = Shape<PREC>;
    using UT = typename std::conditional<PREC == 64, double, float>::type;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double s_val[4], s_part[2];
    __shared__ int s_ok, s_stop;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, nblk = gridDim.x, blk = blockIdx.x;
    unsigned char *scratch = smem + (size_t)Sh::W * Sh::S * Sh::stage;
    double *sh = reinterpret_cast<double *>(scratch);   // two rows of kResThreads
    if (t == 0) {
        s_stop = a.st->stop;
        s_ok = 1;
    }
    __syncthreads();
    if (s_stop) return;   // read once per block, before any block writes it
    double up = a.st->up;
    const double ff = a.st->ff, tol = a.st->tol;
    int iters = a.st->iters;
    const int limit = a.st->limit;
    const double root_ff = CHECON ? 0.0 : sqrt(ff), stop_rr = stop_square(tol, root_ff);
    unsigned long long target = 0;   // arrivals that complete the next exchange
    double *p_pu = a.part, *p_rd = p_pu + kMaxBlocks, *p_2 = p_rd + kMaxBlocks, *p_3 = p_2 + kMaxBlocks;

    // elements of this warp
    const int per_el = (a.nels + nblk - 1) / nblk;
    const int e1 = min(a.nels, (blk + 1) * per_el), first = blk * per_el + w;
    const int nmine = w < Sh::W && first < e1 ? (e1 - first + Sh::W - 1) / Sh::W : 0;
    const bool resident = nmine <= Sh::S || (PREC == 64 && a.stride == 0);
    unsigned char *stage = smem + (size_t)(w < Sh::W ? w : 0) * Sh::S * Sh::stage;
    unsigned char *pw = scratch + (size_t)(w < Sh::W ? w : 0) * Sh::pbytes;
    uint64_t *bar = reinterpret_cast<uint64_t *>(scratch + kScratch<PREC>) + 3 * (w < Sh::W ? w : 0);
    const uint64_t pol = tc::l2_evict_first_policy();
    // ring slot c: chunk c of a record (FP64, one stage) or stage c
    auto issue = [&](int c, int k) {
        const size_t e = (size_t)first + (size_t)k * Sh::W;
        if constexpr (PREC == 64) {
            tc::mbar_expect_tx(&bar[c], fx::chunk_bytes(c));
            tc::bulk_g2s_hint(stage + c * fx::kChunk0, a.rec + e * a.stride + fx::chunk_off(c), fx::chunk_bytes(c), &bar[c],
                              pol);
        } else {
            tc::mbar_expect_tx(&bar[c], Sh::rec);
            tc::bulk_g2s_hint(stage + c * Sh::stage, a.rec + e * a.stride, Sh::rec, &bar[c], pol);
        }
    };
    if (nmine > 0) {
        if (lane == 0) {
            for (int c = 0; c < 3; ++c) tc::mbar_init(&bar[c], 1);
            tc::mbar_fence_init();
        }
        __syncwarp();
        if (lane == 0)
            for (int c = 0; c < (PREC == 64 ? 3 : Sh::S); ++c)
                if (PREC == 64 || c < nmine) issue(c, PREC == 64 ? 0 : c);
    }
    auto node = [&](int k) { return lane < 20 && nmine > 0 ? a.conn[((size_t)first + (size_t)(k % nmine) * Sh::W) * 20 + lane] : 0; };
    const int nd0 = node(0), nd1 = node(1);
    // this lane's two freedoms of an element: rows 2l, 2l+1 (FP64) or l, l+30
    const int l30 = lane < 30 ? lane : 29;
    const int ja = PREC == 64 ? 2 * l30 : l30, jb = PREC == 64 ? 2 * l30 + 1 : l30 + 30;
    bool start = true;   // p is complete in memory; later p = d + beta p
    double beta = 0.0;
    auto gather = [&](int nd, double &va, double &vb) {
        const int na = __shfl_sync(FULLMASK, nd, ja / 3), nb = __shfl_sync(FULLMASK, nd, jb / 3);
        const size_t oa = (size_t)3 * na + ja % 3, ob = (size_t)3 * nb + jb % 3;
        va = __ldcg(a.p + oa);
        vb = __ldcg(a.p + ob);
        if (!start) {
            va = fma(va, beta, __ldcg(a.d + oa));
            vb = fma(vb, beta, __ldcg(a.d + ob));
        }
        if (PREC != 64 && lane >= 30) va = vb = 0.0;   // put_p's means are sums over all lanes
    };

    // slots of this thread
    const int s0 = blk * a.per_slots, s1 = min(a.ns, s0 + a.per_slots);
    const int nact = min(kResThreads, a.per_slots), nwact = (nact + 31) >> 5;   // threads and warps with slots
    auto block_total = [&](int row) {   // by warp `row`, over the warps with slots
        double s = sh[row * kResThreads + lane];
        for (int j = 1; j < nwact; ++j) s += sh[row * kResThreads + lane + 32 * j];
        return warp_sum(s);
    };
    auto meet = [&]() {   // by one thread, after all have raised target
        if (exchange(a.count, target)) return;
        s_ok = 0;
        atomicExch(a.kerr, 3);
        atomicExch(&a.st->stop, 1);
    };

    bool failed = false;
    unsigned g = 0;   // elements this warp has multiplied (ring position)
    double pc[NSL], uu[NSL];
    int it = 0;
    bool stop = false;
    for (; it < a.niters && !stop; ++it) {
        // ---- elements
        double pu = 0.0;
        if (nmine > 0) {
            double pa, pb;
            gather(nd0, pa, pb);
            int nd = nd1;
            for (int k = 0; k < nmine; ++k, ++g) {
                double na = 0.0, nb = 0.0;
                if (k + 1 < nmine) {
                    gather(nd, na, nb);
                    nd = node(k + 2);
                }
                const size_t e = (size_t)first + (size_t)k * Sh::W;
                if constexpr (PREC == 64) {
                    double u0, u1;
                    const bool ok = fx::product(
                        lane, pa, pb, reinterpret_cast<int4 *>(pw),
                        [&](int c) -> const unsigned char * {
                            const uint32_t par = resident ? 0u : (g & 1u);
                            return __all_sync(FULLMASK, tc::mbar_wait(&bar[c], par)) ? stage + c * fx::kChunk0 : nullptr;
                        },
                        [&](int c) {
                            __syncwarp();
                            if (!resident && lane == 0) {
                                tc::fence_proxy_async();
                                issue(c, (k + 1) % nmine);
                            }
                        },
                        u0, u1);
                    if (!ok) {
                        failed = true;
                        break;
                    }
                    if (lane < 30) {
                        reinterpret_cast<double2 *>((double *)a.ut + e * 60)[lane] = make_double2(u0, u1);
                        pu = fma(pa, u0, pu);
                        pu = fma(pb, u1, pu);
                    }
                } else {
                    const int c = resident ? k : (int)(g % Sh::S);
                    const uint32_t par = resident ? 0u : ((g / Sh::S) & 1u);
                    float *pp = reinterpret_cast<float *>(pw);
                    sym::put_p<PREC == 16>(lane, pa, pb, pp);
                    if (!__all_sync(FULLMASK, tc::mbar_wait(&bar[c], par))) {
                        failed = true;
                        break;
                    }
                    __syncwarp();
                    float ra, rb;
                    if constexpr (PREC == 32)
                        sym::walk32(lane, reinterpret_cast<const float *>(stage + c * Sh::stage), pp, ra, rb);
                    else
                        sym::walk16(lane, reinterpret_cast<const uint32_t *>(stage + c * Sh::stage), pp, ra, rb);
                    sym::project_result(lane, ra, rb);
                    if (lane < 30) {
                        float *o = (float *)a.ut + e * 80;
                        o[(lane / 3) * 4 + lane % 3] = ra;
                        o[(lane / 3 + 10) * 4 + lane % 3] = rb;
                        pu = fma(pa, (double)ra, pu);
                        pu = fma(pb, (double)rb, pu);
                    }
                    __syncwarp();
                    if (!resident && lane == 0) {
                        tc::fence_proxy_async();
                        issue(c, (k + Sh::S) % nmine);
                    }
                }
                pa = na;
                pb = nb;
            }
            if (failed && lane == 0) {
                atomicExch(a.kerr, 2);
                atomicExch(&a.st->stop, 1);
                s_ok = 0;
            }
        }
        if (w < Sh::W) reinterpret_cast<double *>(pw)[lane] = pu;   // the warp's p words are free
        target += nblk;
        __syncthreads();
        if (!s_ok) break;
        if (w == kResThreads / 32 - 1) {   // a warp of its own: the others load meanwhile
            double mine = 0.0;
#pragma unroll
            for (int j = 0; j < Sh::W; ++j) mine += reinterpret_cast<const double *>(scratch + j * Sh::pbytes)[lane];
            mine = warp_sum(mine);
            if (lane == 0) {
                p_pu[blk] = mine;
                meet();
            }
            __syncwarp();
        }
        // the owners' p, while the flags travel
        int k0[NSL], k1[NSL];
#pragma unroll
        for (int i = 0; i < NSL; ++i) {
            const int s = s0 + t + i * kResThreads;
            pc[i] = 0.0;
            k0[i] = k1[i] = 0;
            if (s < s1) {
                pc[i] = a.p[s];
                if (!start) pc[i] = fma(pc[i], beta, a.d[s]);
                k0[i] = __ldg(a.ptr + s / 3);
                k1[i] = (__ldg(a.fm + s / 3) >> (s % 3)) & 1 ? __ldg(a.ptr + s / 3 + 1) : k0[i];   // restrained: u = 0
            }
        }
        __syncthreads();
        if (!s_ok) break;
        // ---- slots; the step length meanwhile, by the warp that met
        if (w == kResThreads / 32 - 1) {
            const double sum = add_shares(p_pu, nblk, lane);
            if (lane == 0) s_val[0] = up / sum;
        }
        double xo[NSL], ro[NSL], dv[NSL];
#pragma unroll
        for (int i = 0; i < NSL; ++i) {
            const int s = s0 + t + i * kResThreads;
            uu[i] = xo[i] = ro[i] = dv[i] = 0.0;
            if (s < s1) {
                const int dof = s % 3;
                xo[i] = a.x[s];
                ro[i] = a.r[s];
                dv[i] = __ldg(a.dinv + s);
                UT acc = 0;
                for (int k = k0[i]; k < k1[i]; k += 4) {   // four contributions in flight, added in order
                    UT v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int ci = k + q < k1[i] ? __ldg(a.list + k + q) : -1;
                        v[q] = ci < 0 ? (UT)0
                               : PREC == 64 ? (UT)__ldcg((const double *)a.ut + (size_t)ci * 3 + dof)
                                            : (UT)__ldcg((const float *)a.ut + (size_t)ci * 4 + dof);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (k + q < k1[i]) acc += v[q];
                }
                uu[i] = (double)acc;
                a.p[s] = pc[i];   // every gather of the old p is behind the flags
            }
        }
        __syncthreads();
        const double alpha = s_val[0];
        double rd = 0.0, rr = 0.0;
        long long mx = 0, md = 0;
#pragma unroll
        for (int i = 0; i < NSL; ++i) {
            const int s = s0 + t + i * kResThreads;
            if (s < s1) {
                const double xn = fma(pc[i], alpha, xo[i]);
                a.x[s] = xn;
                if (CHECON) {
                    mx = max(mx, abs_bits(xn));
                    md = max(md, abs_bits(xn - xo[i]));
                }
                const double rn = fma(-uu[i], alpha, ro[i]), dn = dv[i] * rn;
                a.r[s] = rn;
                a.d[s] = dn;
                rd = fma(rn, dn, rd);
                if (!CHECON) rr = fma(rn, rn, rr);
            }
        }
        sh[t] = rd;
        if (!CHECON) sh[kResThreads + t] = rr;
        if (CHECON) block_max2(mx, md);   // (its barriers order sh too)
        __syncthreads();
        if (w == 0 || (w == 1 && !CHECON)) {
            const double mine = block_total(w);
            if (lane == 0) s_part[w] = mine;
        }
        target += nblk;
        __syncthreads();
        if (t == 0) {
            p_rd[blk] = s_part[0];
            p_2[blk] = CHECON ? __longlong_as_double(mx) : s_part[1];
            if (CHECON) p_3[blk] = __longlong_as_double(md);
            meet();
        }
        __syncthreads();
        if (!s_ok) break;
        if (w == 2) {   // beta and the stopping value side by side (warp 0, fresh from its wait, takes 0.8 us longer)
            const double sum = add_shares(p_rd, nblk, lane);
            if (lane == 0) {
                s_val[1] = sum;
                s_val[2] = sum / up;
            }
        } else if (w == 1 && CHECON) {
            const long long m = max_shares(p_2, nblk, lane), q = max_shares(p_3, nblk, lane);
            if (lane == 0) {
                s_val[3] = __longlong_as_double(q) / __longlong_as_double(m);   // checon_par's measure
                s_stop = isfinite(__longlong_as_double(m)) ? 0 : 1;
            }
        } else if (w == 1) {
            const double sum = add_shares(p_2, nblk, lane);
            if (lane == 0) {
                s_val[3] = sum;
                s_stop = 0;
            }
        }
        __syncthreads();
        const double rdn = s_val[1], measure = s_val[3];
        beta = s_val[2];
        ++iters;
        // ||r|| / ||f|| <= tol as r.r <= (tol ||f||)^2: two roots and a
        // division would be a tenth of the iteration
        const bool conv = CHECON ? measure <= tol : measure <= stop_rr;
        const bool bad = !isfinite(rdn) || s_stop != 0;
        stop = conv || iters >= limit || bad;
        if (blk == 0 && t == 0 && (stop || it + 1 == a.niters)) {
            volatile PcgState *vs = a.st;
            vs->up = rdn;
            vs->beta = beta;
            vs->iters = iters;
            vs->rr = CHECON ? 0.0 : measure;
            vs->metric = CHECON ? measure : sqrt(measure) / root_ff;
            vs->converged = conv ? 1 : 0;
            if (bad) vs->err = 1;
            if (stop) vs->stop = vs->stop2 = 1;
        }
        up = rdn;
        start = false;
    }
    // p of the next iteration, as update2 leaves it
    if (s_ok && !start) {
#pragma unroll
        for (int i = 0; i < NSL; ++i) {
            const int s = s0 + t + i * kResThreads;
            if (s < s1) a.p[s] = fma(pc[i], beta, a.d[s]);
        }
    }
    // wait (bounded) for the copies this warp still has in flight: the ring's
    // next ones, or, when a wait ran out, whatever had been issued
    if (nmine > 0 && (!resident || failed)) {
        if constexpr (PREC == 64) {
            for (int c = 0; c < 3; ++c) {
                tc::mbar_wait(&bar[c], resident ? 0u : g & 1u);
                if (failed && !resident) tc::mbar_wait(&bar[c], (g + 1) & 1u);
            }
        } else {
            for (unsigned q = g; q < g + Sh::S; ++q)
                if (!resident || (int)(q - g) < nmine) tc::mbar_wait(&bar[q % Sh::S], resident ? 0u : (q / Sh::S) & 1u);
        }
    }
}

// ---------------------------------------------------------------------------
// Rule: 20-node meshes with records (one per element, or FP64 one for all)
// whose slots fit the CTAs, four per thread (311,296 on 152 SMs: 28^3 elements).  Measured us per
// iteration, this kernel / four kernels in a graph:
//            10^3        16^3        20^3        24^3        28^3
//   FP64     10.8/21.5   22.0/30.5   36.1/43.4   56.0/63.1   82.0/87.0
//   FP32     11.4/22.7   15.7/28.8   24.3/33.0   34.3/43.8   46.1/56.8
//   FP16     10.1/22.2   13.7/24.5   22.7/29.0   29.9/35.5   40.9/45.8
// so that it takes every mesh that fits.  Of the 10.8 us at 10^3 (FP64)
// the products take 3.8, the two exchanges 2.6 and the sums over the CTAs with
// the two divisions 2.5.
//
// The kernel holds its SMs for the whole run, so that runs of other contexts
// wait for it.  Meshes whose products lose nothing by it take half the SMs,
// and two such runs go side by side: those of at most so many elements per
// CTA, in FP64 three (they share the SM's integer pipe), in FP32 ten, in FP16
// seven.  us per iteration on all SMs / on half (one context's spread by where
// its counter lies is 4 %, but these are of the same contexts):
//            6^3          4 x 8 x 7    7^3          8^3          9^3          10^3
//   FP64     11.1/10.5    11.0/10.4    11.5/11.5    10.6/11.6    11.3/12.4    11.5/13.6
//   FP32     13.0/12.5    12.5/11.6    12.6/12.9    12.7/12.4    12.5/12.5    12.9/13.1
//   FP16     12.7/12.2    12.2/11.4    12.5/12.2    11.7/11.7    11.5/11.7    11.6/12.1
// and solves per second of eight contexts in threads, all / half / the separate
// kernels that have no such runs: 6^3 FP64 716/1432/1333, FP32 612/1250/876,
// 9^3 FP32 413/798/669, 8^3 FP16 510/996/785; where all SMs are kept, 8^3 FP64
// 565/1044/789, 10^3 FP32 356/681/508, FP16 407/766/494.
// (The number of CTAs must not depend on what else runs: it orders the sums.)
static int resident_ctas(const Ctx &c, int prec)
{
    const int half = c.nsm / 2, per = prec == PREC_FP64 ? 3 : prec == PREC_FP32_SYM ? 10 : 7;
    return half > 0 && c.nels <= per * half ? half : c.nsm;
}
static int slots_per_block(const Ctx &c, int ctas) { return (c.nslots + ctas - 1) / ctas; }

bool resident_ok(const Ctx &c, int prec)
{
    if (c.kind != KIND_SOLID20 || c.nsm > kMaxBlocks || c.no_coop) return false;
    if (slots_per_block(c, resident_ctas(c, prec)) > 4 * kResThreads) return false;
    if (c.shared) return prec == PREC_FP64 && c.skmfix;
    return prec == PREC_FP64 ? c.kmfix != nullptr : prec == PREC_FP32_SYM || prec == PREC_FP16_SYM;
}

// The result of a cooperative launch that failed with e
static int coop_failed(Ctx &c, const char *name, cudaError_t e)
{
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported) {
        cudaGetLastError();
        c.no_coop = true;
        return kRefused;
    }
    set_error("%s: cooperative launch of %d blocks failed: %s", name, c.nsm, cudaGetErrorString(e));
    return 1;
}

template <int PREC, bool CHECON, int NSL>
static int launch_resident_t(Ctx &c, double *xsol, int niters, int ctas)
{
    constexpr size_t smem = kResSmem<PREC>;
    static_assert(smem + 256 + 2 * 32 * 8 <= 227 * 1024, "shared memory per CTA");
    const void *fn = (const void *)k_pcg_resident<PREC, CHECON, NSL>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    ResArgs a;
    a.nels = c.nels;
    a.ns = c.nslots;
    a.niters = niters;
    a.per_slots = slots_per_block(c, ctas);
    a.stride = c.shared ? 0 : Shape<PREC>::rec;
    a.rec = c.shared ? c.skmfix : PREC == 64 ? c.kmfix : PREC == 32 ? (const unsigned char *)c.km32p : (const unsigned char *)c.km16p;
    a.conn = c.conn;
    a.ut = c.utemp;
    a.ptr = c.node_ptr;
    a.list = c.node_list;
    a.fm = c.freemask;
    a.x = xsol;
    a.r = c.r;
    a.d = c.d;
    a.p = c.p;
    a.dinv = c.dinv;
    a.st = c.st;
    a.count = reinterpret_cast<unsigned long long *>(c.res_part);
    a.part = c.res_part + 8;
    if (e == cudaSuccess) e = cudaMemsetAsync(a.count, 0, sizeof(unsigned long long), c.stream);
    a.kerr = c.kerr;
    void *args[] = {&a};
    if (e == cudaSuccess) e = cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(kResThreads), args, smem, c.stream);
    if (e != cudaSuccess) return coop_failed(c, "k_pcg_resident", e);
    c.launches++;
    return 0;
}

template <int PREC>
static int launch_resident_p(Ctx &c, double *xsol, int niters)
{
    const int n = resident_ctas(c, PREC);
    const bool ck = c.stop_mode == STOP_CHECON, one = slots_per_block(c, n) <= kResThreads;
    if (PREC == 64 && ck)   // checon_par stops FP64 runs only
        return one ? launch_resident_t<PREC, PREC == 64, 1>(c, xsol, niters, n)
                   : launch_resident_t<PREC, PREC == 64, 4>(c, xsol, niters, n);
    return one ? launch_resident_t<PREC, false, 1>(c, xsol, niters, n) : launch_resident_t<PREC, false, 4>(c, xsol, niters, n);
}

int launch_pcg_resident(Ctx &c, int prec, double *xsol, int niters)
{
    return prec == PREC_FP64 ? launch_resident_p<64>(c, xsol, niters)
           : prec == PREC_FP32_SYM ? launch_resident_p<32>(c, xsol, niters)
                                   : launch_resident_p<16>(c, xsol, niters);
}

// ---------------------------------------------------------------------------
// The rest of an iteration behind the element products, in one cooperative
// launch, for meshes that the resident kernel does not take: one CTA of 1024
// threads per SM, which keeps u and then d of its slots in shared memory (7 of
// the 13 vector streams of the separate kernels are left), and two exchanges
// where they have launches.  Node sums go a thread per node (one 16-byte load
// per FP32 contribution), everything else a thread per slot: sums per slot
// took 162 instead of 152 us of a 64^3 iteration with one element matrix.
// Bound by the chain of sums, exchange and division at 33^3 (a third of it)
// and by the FP64 pipe (eight operations per slot, two per SM and clock: 45
// us at 64^3) and memory (270 MB, 40 us) together at 64^3, 80 us in all.
// More loads in flight do not help: L2 prefetches of the next 32 nodes'
// vectors and results took 394 and 405 instead of 392 us per iteration.
constexpr int kTailThreads = 1024;

struct TailArgs {
    int nn, per_nodes, ns;       // GIVEN: nodes of three slots each, in name only
    const void *ut;
    const int *ptr, *list;
    const uint8_t *fm;
    double *x, *r, *p;
    const double *dinv, *u;
    float2 *ps;                  // the FP32 parts of p (shared km), or null
    PcgState *st;
    unsigned long long *count;   // arrivals, zeroed by launch_pcg_init
    double *part;
    const double *pu;            // [npu] the products' shares of p.u (DOT)
    int npu;
    const unsigned char *rec;    // the next products' records, `ahead` of each of their CTAs to be fetched into L2
    int rec_bytes, nels, per_el, ahead;
    int *kerr;
};

// One warp: the sum over a block's threads, in four chains per lane
__device__ __forceinline__ double tail_total(const double *sh, int lane)
{
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[q] = sh[lane + 32 * q];
#pragma unroll
        for (int j = 1; j < kTailThreads / 128; ++j) v[q] += sh[lane + 32 * q + 128 * j];
    }
    return warp_sum((v[0] + v[1]) + (v[2] + v[3]));
}

// A warp goes through its nodes 32 at a time, sums by node and the rest by
// slot: 96 slots, which change lanes through su.  DOT: the products' CTAs
// have left their shares of p.u, so that alpha is known at once and the node
// sums (latency) run together with x, r and d (the FP64 pipe).  Otherwise
// p.u is formed here, behind an exchange.
// GIVEN (8-node meshes): the product kernel has left u and alpha.
enum { TAIL_SUMS = 0, TAIL_DOT = 1, TAIL_GIVEN = 2 };
template <typename UT, bool CHECON, int HOW>
__global__ void __launch_bounds__(kTailThreads, 1) k_pcg_tail(TailArgs a)
{
    extern __shared__ double su[];   // u, then d, of the block's slots
    __shared__ double sh[2][kTailThreads];
    __shared__ double s_val[4], s_part[2], s_bound;
    __shared__ int s_ok, s_stop;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, nblk = gridDim.x, blk = blockIdx.x;
    if (t == 0) {
        s_stop = a.st->stop;
        s_ok = 1;
    }
    __syncthreads();
    if (s_stop) return;   // read once per block, before any block writes it
    const double up = a.st->up, tol = a.st->tol;
    const int iters = a.st->iters;
    unsigned long long target = ((HOW == TAIL_SUMS ? 2ULL : 1ULL) * iters + 1) * nblk;   // arrivals that complete the next exchange
    double *p_pu = a.part, *p_rd = p_pu + kMaxBlocks, *p_2 = p_rd + kMaxBlocks, *p_3 = p_2 + kMaxBlocks;
    auto meet = [&]() {
        if (exchange(a.count, target)) return;
        s_ok = 0;
        atomicExch(a.kerr, 3);
        atomicExch(&a.st->stop, 1);
    };
    // this warp's nodes: 32 from node c on, then from c + kTailThreads on, ...
    const int n0 = blk * a.per_nodes, n1 = min(a.nn, n0 + a.per_nodes), s0 = 3 * n0, s1 = min(a.ns, 3 * n1), c0 = n0 + 32 * w;
    // ---- sums over a node's elements (ascending) into su
    auto node_sums = [&](int n) {
        const int k1 = __ldg(a.ptr + n + 1), m = __ldg(a.fm + n);
        UT u0 = 0, u1 = 0, u2 = 0;
        for (int k = __ldg(a.ptr + n); k < k1; k += 4) {   // four contributions in flight
            int ci[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) ci[q] = __ldg(a.list + min(k + q, k1 - 1));
            UT v[4][3];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if constexpr (sizeof(UT) == 4) {
                    const float4 f = __ldg((const float4 *)a.ut + ci[q]);
                    v[q][0] = f.x;
                    v[q][1] = f.y;
                    v[q][2] = f.z;
                } else {
#pragma unroll
                    for (int d = 0; d < 3; ++d) v[q][d] = __ldg((const double *)a.ut + (size_t)ci[q] * 3 + d);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (k + q < k1) {
                    u0 += v[q][0];
                    u1 += v[q][1];
                    u2 += v[q][2];
                }
        }
        double *o = su + 3 * (n - n0);
        o[0] = m & 1 ? (double)u0 : 0.0;   // restrained: u = 0
        o[1] = m & 2 ? (double)u1 : 0.0;
        o[2] = m & 4 ? (double)u2 : 0.0;
    };
    // ---- x, r, d of the 96 slots of 32 nodes
    double alpha = 0.0, rd = 0.0, rr = 0.0;
    long long mx = 0, md = 0;
    double xo[3], ro[3], dv[3], po[3];
    auto fetch = [&](int c) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int s = 3 * c + lane + 32 * j;
            if (s < s1) {
                po[j] = a.p[s];
                xo[j] = a.x[s];
                ro[j] = a.r[s];
                dv[j] = __ldg(a.dinv + s);
                if (HOW == TAIL_GIVEN) su[s - s0] = a.u[s];
            }
        }
    };
    auto step = [&](int c) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int s = 3 * c + lane + 32 * j;
            if (s < s1) {
                const double xn = fma(po[j], alpha, xo[j]);
                a.x[s] = xn;
                if (CHECON) {
                    mx = max(mx, abs_bits(xn));
                    md = max(md, abs_bits(xn - xo[j]));
                }
                const double rn = fma(-su[s - s0], alpha, ro[j]), dn = dv[j] * rn;
                a.r[s] = rn;
                su[s - s0] = dn;
                rd = fma(rn, dn, rd);
                if (!CHECON) rr = fma(rn, rn, rr);
            }
        }
    };
    if (w == 1 && !CHECON && lane == 0) s_bound = stop_square(tol, sqrt(a.st->ff));
    if (HOW == TAIL_GIVEN) {
        alpha = a.st->alpha;
        for (int c = c0; c < n1; c += kTailThreads) {
            fetch(c);
            step(c);
        }
    } else if (HOW == TAIL_DOT) {
        if (c0 < n1) fetch(c0);
        if (w == kTailThreads / 32 - 1) {   // it has its sums when the others have theirs
            const double sum = add_shares(a.pu, a.npu, lane);
            if (lane == 0) s_val[0] = up / sum;
        }
        if (c0 + lane < n1) node_sums(c0 + lane);
        __syncthreads();
        alpha = s_val[0];
        for (int c = c0; c < n1;) {
            step(c);
            c += kTailThreads;
            if (c < n1) {
                fetch(c);
                if (c + lane < n1) node_sums(c + lane);
                __syncwarp();
            }
        }
    } else {
        double pu = 0.0;
        for (int c = c0; c < n1; c += kTailThreads) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int s = 3 * c + lane + 32 * j;
                po[j] = s < s1 ? a.p[s] : 0.0;
            }
            if (c + lane < n1) node_sums(c + lane);
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int s = 3 * c + lane + 32 * j;
                if (s < s1) pu = fma(po[j], su[s - s0], pu);
            }
        }
        sh[0][t] = pu;
        if (c0 < n1) fetch(c0);
        __syncthreads();
        if (w == 0) {
            const double mine = tail_total(sh[0], lane);
            if (lane == 0) {
                p_pu[blk] = mine;
                meet();
            }
            __syncwarp();
            const double sum = add_shares(p_pu, nblk, lane);
            if (lane == 0) s_val[0] = up / sum;
        }
        target += nblk;
        __syncthreads();
        if (!s_ok) return;
        alpha = s_val[0];
        for (int c = c0; c < n1;) {
            step(c);
            c += kTailThreads;
            if (c < n1) fetch(c);
        }
    }
    sh[0][t] = rd;
    if (!CHECON) sh[1][t] = rr;
    if (CHECON) block_max2(mx, md);
    // the next products' first records on their way to L2
    if (t < a.ahead && blk * a.per_el + t < min(a.nels, (blk + 1) * a.per_el))
        tc::bulk_prefetch(a.rec + (size_t)(blk * a.per_el + t) * a.rec_bytes, a.rec_bytes);
    // p of the first slots, in flight beside the sums
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const int s = 3 * c0 + lane + 32 * j;
        po[j] = s < s1 ? a.p[s] : 0.0;
    }
    __syncthreads();
    if (w == 0 || (w == 1 && !CHECON)) {
        const double mine = tail_total(sh[w], lane);
        if (lane == 0) s_part[w] = mine;
    }
    __syncthreads();
    if (t == 0) {
        p_rd[blk] = s_part[0];
        p_2[blk] = CHECON ? __longlong_as_double(mx) : s_part[1];
        if (CHECON) p_3[blk] = __longlong_as_double(md);
        meet();
    }
    __syncthreads();
    if (!s_ok) return;
    if (w == 2) {
        const double sum = add_shares(p_rd, nblk, lane);
        if (lane == 0) {
            s_val[1] = sum;
            s_val[2] = sum / up;
        }
    } else if (w == 1 && blk == 0) {   // the stopping test is block 0's
        if (CHECON) {
            const long long m = max_shares(p_2, nblk, lane), q = max_shares(p_3, nblk, lane);
            if (lane == 0) {
                s_val[3] = __longlong_as_double(q) / __longlong_as_double(m);   // checon_par's measure
                s_stop = isfinite(__longlong_as_double(m)) ? 0 : 1;
            }
        } else {
            const double sum = add_shares(p_2, nblk, lane);
            if (lane == 0) s_val[3] = sum;
        }
    }
    __syncthreads();
    // ---- p
    const double beta = s_val[2];
    for (int c = c0; c < n1;) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int s = 3 * c + lane + 32 * j;
            if (s < s1) {
                const double pn = fma(po[j], beta, su[s - s0]);
                a.p[s] = pn;
                if (a.ps) {
                    float h, l;
                    tc::split_f64(pn, h, l);
                    a.ps[s] = make_float2(h, l);
                }
            }
        }
        c += kTailThreads;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int s = 3 * c + lane + 32 * j;
            po[j] = s < s1 ? a.p[s] : 0.0;
        }
    }
    if (blk == 0 && t == 0) {
        const double rdn = s_val[1], measure = s_val[3];
        const bool conv = CHECON ? measure <= tol : measure <= s_bound;
        const bool bad = !isfinite(rdn) || s_stop != 0;
        volatile PcgState *vs = a.st;
        vs->up = rdn;
        vs->beta = beta;
        vs->iters = iters + 1;
        vs->rr = CHECON ? 0.0 : measure;
        vs->converged = conv ? 1 : 0;
        if (bad) vs->err = 1;
        if (conv || iters + 1 >= vs->limit || bad) {   // two roots and a division: only when they are read
            vs->metric = CHECON ? measure : sqrt(measure) / sqrt(vs->ff);
            vs->stop = vs->stop2 = 1;
        }
    }
}

// Bytes of records per CTA fetched into L2 while the sums cross the chip:
// the next products start from L2 instead of HBM.  us per iteration with
// and without: 31^3 FP64 99.3/104.9, FP32 55.2/57.9, FP16 44.9/47.6; 36^3 146.3/147.3, 77.5/79.2, 59.8/61.0;
// 45^3 and larger within 1 %.  More (120, 240 KB), or at the start of the
// tail, is in the way of its own loads (31^3 120 MB: 108, 65.6, 51.2 us).
constexpr int kAheadBytes = 60 << 10;

constexpr int kTailMax = 26;   // slots per thread that fit in shared memory

// Rule: meshes whose slots fit the CTAs' shared memory (4,046,848 on 152
// SMs).  us per iteration with this kernel / with scatter, update1 and
// update2 in a graph:
//                          33^3          45^3        55^3        64^3
//   FP64                   121/125       278/288     491/502     771/782
//   FP32                   65/74         145/162     251/263     392/409
//   FP16                   52/59         104/117     172/182     270/273
//   FP32, one matrix       36/43         61/74       93/103      148/153
// 8-node meshes (two updates before): p123 32^3 18.9/20.3, 50^3 26.8/30.4,
// 100^3 92/95; below 30,000 slots (24^3: 19.4/17.4) two dependent launches
// cost less than an exchange.
static int tail_nodes(const Ctx &c) { return ((c.nslots + 2) / 3 + c.nsm - 1) / c.nsm; }

bool tail_ok(const Ctx &c)
{
    if (c.no_coop) return false;
    if (c.kind != KIND_SOLID20 && c.nslots < 30000) return false;
    return c.nsm <= kMaxBlocks && 3 * tail_nodes(c) <= kTailMax * kTailThreads;
}

// The shared memory of the tail's largest form (outside any stream capture)
int prepare_tail(Ctx &c)
{
    if (c.tail_attr) return 0;
    const void *fn[] = {(const void *)k_pcg_tail<double, true, TAIL_SUMS>, (const void *)k_pcg_tail<double, false, TAIL_SUMS>,
                        (const void *)k_pcg_tail<float, false, TAIL_SUMS>, (const void *)k_pcg_tail<float, false, TAIL_DOT>,
                        (const void *)k_pcg_tail<double, true, TAIL_GIVEN>, (const void *)k_pcg_tail<double, false, TAIL_GIVEN>};
    for (const void *f : fn) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   kTailMax * kTailThreads * (int)sizeof(double));
        if (e != cudaSuccess) {
            set_error("k_pcg_tail: cannot reserve shared memory: %s", cudaGetErrorString(e));
            return 1;
        }
    }
    c.tail_attr = true;
    return 0;
}

// The records that the next products read first
static void records_ahead(const Ctx &c, int prec, TailArgs &a)
{
    a.nels = c.nels;
    a.per_el = (c.nels + element_ctas(c) - 1) / element_ctas(c);
    a.ahead = 0;
    a.rec = nullptr;
    a.rec_bytes = 0;
    if (c.kind != KIND_SOLID20 || c.shared) return;
    if (prec == PREC_FP64 && c.kmfix) {
        a.rec = c.kmfix;
        a.rec_bytes = fx::kRecBytes;
    } else if (prec == PREC_FP32_SYM) {
        a.rec = (const unsigned char *)c.km32p;
        a.rec_bytes = sym::kBytes32;
    } else if (prec == PREC_FP16_SYM) {
        a.rec = (const unsigned char *)c.km16p;
        a.rec_bytes = sym::kBytes16;
    } else {
        return;
    }
    a.ahead = kAheadBytes / a.rec_bytes;
}

template <typename UT, bool CHECON, int HOW>
static int launch_tail_t(Ctx &c, int prec, double *xsol, int npu)
{
    TailArgs a;
    records_ahead(c, prec, a);
    a.nn = (c.nslots + 2) / 3;
    a.per_nodes = tail_nodes(c);
    a.ns = c.nslots;
    a.u = c.u;
    a.ut = c.utemp;
    a.ptr = c.node_ptr;
    a.list = c.node_list;
    a.fm = c.freemask;
    a.x = xsol;
    a.r = c.r;
    a.p = c.p;
    a.dinv = c.dinv;
    a.ps = c.shared ? c.psplit : nullptr;
    a.st = c.st;
    a.count = c.gbar + kTailBar * kBarWords;
    a.part = c.res_part + 8;
    a.pu = c.res_part + 8 + 4 * kMaxBlocks;
    a.npu = npu;
    a.kerr = c.kerr;
    const size_t smem = (size_t)a.per_nodes * 3 * sizeof(double);
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_pcg_tail<UT, CHECON, HOW>, dim3(c.nsm),
                                                      dim3(kTailThreads), args, smem, c.stream);
    if (e != cudaSuccess) return coop_failed(c, "k_pcg_tail", e);
    c.launches++;
    return 0;
}

int launch_iteration_tail(Ctx &c, int prec, double *xsol, int npu)
{
    const bool ck = c.stop_mode == STOP_CHECON;   // FP64 runs only
    if (c.kind != KIND_SOLID20)
        return ck ? launch_tail_t<double, true, TAIL_GIVEN>(c, prec, xsol, 0) : launch_tail_t<double, false, TAIL_GIVEN>(c, prec, xsol, 0);
    if (prec == PREC_FP64)
        return ck ? launch_tail_t<double, true, TAIL_SUMS>(c, prec, xsol, 0) : launch_tail_t<double, false, TAIL_SUMS>(c, prec, xsol, 0);
    return npu ? launch_tail_t<float, false, TAIL_DOT>(c, prec, xsol, npu) : launch_tail_t<float, false, TAIL_SUMS>(c, prec, xsol, 0);
}

// (the resident run zeroes the counter before every launch)
int launch_exchange_probe(Ctx &c, long long polls)
{
    k_exchange_probe<<<1, 32, 0, c.stream>>>(reinterpret_cast<unsigned long long *>(c.res_part), polls, c.kerr);
    c.launches++;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("k_exchange_probe: launch failed: %s", cudaGetErrorString(e));
        return 1;
    }
    return 0;
}

double *product_shares(Ctx &c) { return c.res_part + 8 + 4 * kMaxBlocks; }

}  // namespace pf
