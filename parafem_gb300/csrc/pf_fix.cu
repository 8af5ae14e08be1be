// pf_fix.cu -- FP64 element products in 64-bit fixed point (pf_fix.cuh), and
// the one pass over the FP64 storkm that writes its packed forms.
#include "pf_fix.cuh"
#include "pf_tc.cuh"

namespace pf {

namespace {

constexpr int kPackThreads = 256;
constexpr int kPacked32 = 1832;   // floats per element of the packed FP32 storkm (packed_off)

// entry (i, k) of the 8-byte word pair w of a record, words counted from its
// start: false where a record holds no entry
__device__ __forceinline__ bool word_entry(int w, int &i, int &k)
{
    constexpr int w0 = fx::kOff0 / 8, w11 = fx::kOff11 / 8, w15 = fx::kOff15 / 8, w14 = w15 + 60;
    if (w < w0) return false;
    if (w < w11) {
        i = (w - w0) & ~1;
        k = w - w0;
    } else if (w < w15) {
        i = k = 2 * (w - w11) + 1;
    } else if (w < w14) {
        const int v = w - w15, l = (v % 30) >> 1;
        i = 2 * l + v / 30;
        k = 2 * (l + 15) + (v & 1);
    } else {
        const int v = w - (w < fx::kChunk0 / 8 ? w14 : fx::kChunk0 / 8);
        const int s = (w < fx::kChunk0 / 8 ? 14 : 10) - v / 120, r = v % 120, l = (r % 60) >> 1;
        if (w < fx::kChunk0 / 8 && s < 11) return false;
        i = 2 * l + r / 60;
        k = 2 * (l + s < 30 ? l + s : l + s - 30) + (r & 1);
    }
    return true;
}

}  // namespace

// One block per element (grid-stride): storkm(60,60,e) once through shared
// memory into the packed FP32 diagonals (kp, may be null) and the
// fixed-point record (rec, may be null).  *bad is set when an element is not
// symmetric to the last bit, or an entry does not fit the record (K' not
// below 1, a diagonal that is not positive): the fixed-point form is then
// not used.  An element whose rows of K' sum to less than 15.9 in magnitude
// (a 20-node brick's reach 5 to 9) has room for two more bits per entry.
// Bound by HBM: 28.8 KB read, 7.3 + 14.8 KB written per element.
__global__ void __launch_bounds__(kPackThreads)
k_pack_storkm(int nels, const double *__restrict__ km, float *__restrict__ kp, unsigned char *__restrict__ rec,
              int *__restrict__ bad)
{
    __shared__ __align__(16) double ke[3600];
    __shared__ int sc[60];
    __shared__ int wide;
    const int t = threadIdx.x;
    for (int e = blockIdx.x; e < nels; e += gridDim.x) {
        const double2 *src = reinterpret_cast<const double2 *>(km + (size_t)e * 3600);
        for (int i = t; i < 1800; i += kPackThreads) reinterpret_cast<double2 *>(ke)[i] = __ldcs(src + i);
        if (t == 0) wide = 0;
        __syncthreads();
        bool ok = true;
        unsigned char *out = rec ? rec + (size_t)e * fx::kRecBytes : nullptr;
        if (rec && t < 60) {
            const long long b = __double_as_longlong(ke[61 * t]);
            const int ex = (int)((b >> 52) & 0x7ff);
            ok = b > 0 && ex > 0 && ex < 2047;
            sc[t] = ok ? fx::fix_scale(b) : 0;
            reinterpret_cast<short *>(out + fx::kOffExp)[t] = (short)sc[t];
        }
        if (kp) {
            float *o32 = kp + (size_t)e * kPacked32;
            for (int pos = t; pos < kPacked32; pos += kPackThreads) {
                const int sd = pos < 1800 ? pos / 60 : 30, i = pos - 60 * sd, k = i + sd < 60 ? i + sd : i + sd - 60;
                o32[pos] = pos < 1830 ? (float)ke[60 * k + i] : 0.0f;   // K(i, i+s)
            }
        }
        __syncthreads();
        if (rec) {
            if (t < 240) {   // four threads per row
                const int i = t % 60, q = t / 60;
                int sum = 0;
                for (int k = q; k < 60; k += 4) sum += fx::fix_size(__double_as_longlong(ke[60 * k + i]), sc[i], sc[k]);
                if (sum >= (int)(15.9 / 4 * (1 << 20))) wide = 1;   // each quarter row below 15.9 / 4
            }
            __syncthreads();
            const int extra = wide ? 0 : 2;
            if (t == 0) *reinterpret_cast<int *>(out + fx::kOffExtra) = extra;
            for (int w = t; w < fx::kRecBytes / 8; w += kPackThreads) {
                int i, k;
                if (!word_entry(w, i, k)) continue;
                const long long b = __double_as_longlong(ke[60 * k + i]);
                fx::Words v;
                ok = fx::fix_entry(b, sc[i], sc[k], extra, v) && b == __double_as_longlong(ke[60 * i + k]) && ok;
                reinterpret_cast<int2 *>(out)[w] = make_int2(v.h, v.l);
            }
            if (!ok) atomicOr(bad, 1);
        }
        __syncthreads();
    }
}

// utemp(:,e) = K_e p_e for every element from the fixed-point records.  One
// persistent CTA of 14 warps per SM, one warp per element; each warp streams
// its elements' records through three shared-memory stages (chunk c always
// in stage c) by cp.async.bulk, the next element's chunk issued as soon as
// the warp has read this one's, and gathers p one element ahead.  Every wait
// on an mbarrier is bounded, as in k_elem_sym32.
// Bound by HBM (14,784 B of record + 80 + 480 B per element): 1.30 ms on an
// 80^3 cube, 0.89 of the measured copy bandwidth; the FP64 FMA product of
// the same mesh, k_elem<double>, is bound by the FP64 pipe and takes 3.35 ms
// (40^3: 0.167 against 0.431 ms).  Error against extended precision on
// distorted heterogeneous meshes, 2-norm: 0.2-0.4 of k_elem<double>'s for
// dense p, the same where p has single entries; single rows can be worse
// (pf_fix.cuh, weak_rows).  Loading the blocks
// straight into registers instead of through shared memory took 1.41 ms.
// ROWS: with the rows that FMA holds better formed so from km (weak_rows).
constexpr int kFixWarps = 14;
constexpr size_t kFixSmem = (size_t)kFixWarps * (3 * fx::kChunk0 + 960 + 3 * 8);
static_assert(kFixSmem <= 227 * 1024, "shared memory per CTA");
template <bool ROWS>
__global__ void __launch_bounds__(kFixWarps * 32, 1)
k_elem_fix(int nels, const unsigned char *__restrict__ rec, const int *__restrict__ conn, const double *__restrict__ p,
           double *__restrict__ ut, const PcgState *__restrict__ st, int *__restrict__ err, const double *__restrict__ km)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned char *stage = smem + (size_t)w * 3 * fx::kChunk0;
    int4 *pq = reinterpret_cast<int4 *>(smem + (size_t)kFixWarps * 3 * fx::kChunk0) + w * 60;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + (size_t)kFixWarps * (3 * fx::kChunk0 + 960)) + 3 * w;
    pdl_enter();
    int stopped = 0;
    if (lane == 0 && st) stopped = st->stop;
    if (__shfl_sync(FULLMASK, stopped, 0)) return;
    // this CTA's contiguous element range, warps interleaved inside it
    const int per_cta = (nels + gridDim.x - 1) / gridDim.x;
    const int first = blockIdx.x * per_cta + w, e1 = min(nels, (int)(blockIdx.x + 1) * per_cta);
    if (first >= e1) return;
    const int nmine = (e1 - first + kFixWarps - 1) / kFixWarps;
    if (lane == 0) {
        for (int c = 0; c < 3; ++c) tc::mbar_init(&bar[c], 1);
        tc::mbar_fence_init();
    }
    __syncwarp();
    const uint64_t pol = tc::l2_evict_first_policy();
    auto issue = [&](int c, int k) {   // chunk c of this warp's k-th element (lane 0)
        tc::mbar_expect_tx(&bar[c], fx::chunk_bytes(c));
        tc::bulk_g2s_hint(stage + c * fx::kChunk0, rec + (size_t)(first + k * kFixWarps) * fx::kRecBytes + fx::chunk_off(c),
                          fx::chunk_bytes(c), &bar[c], pol);
    };
    if (lane == 0)
        for (int c = 0; c < 3; ++c) issue(c, 0);
    auto node = [&](int k) { return lane < 20 && k < nmine ? conn[(size_t)(first + k * kFixWarps) * 20 + lane] : 0; };
    int nd = node(0);
    double pa, pb;
    fx::gather2<true>(nd, lane, p, pa, pb);
    nd = node(1);
    int k = 0, chunk = 0;
    bool ok = true;
    for (; k < nmine; ++k) {
        double na, nb, u0, u1;
        bool weak0, weak1;
        fx::gather2<true>(nd, lane, p, na, nb);   // of the next element (of node 0 behind the last)
        nd = node(k + 2);
        ok = fx::product<ROWS>(
            lane, pa, pb, pq,
            [&](int c) -> const unsigned char * {
                chunk = c;
                return __all_sync(FULLMASK, tc::mbar_wait(&bar[c], (uint32_t)(k & 1))) ? stage + c * fx::kChunk0 : nullptr;
            },
            [&](int c) {
                __syncwarp();   // every lane is done with the stage
                if (lane == 0 && k + 1 < nmine) {
                    tc::fence_proxy_async();
                    issue(c, k + 1);
                }
            },
            u0, u1, weak0, weak1);
        if (!ok) break;
        if (ROWS) fx::weak_rows(lane, pa, pb, km + (size_t)(first + k * kFixWarps) * 3600, weak0, weak1, u0, u1);
        if (lane < 30) reinterpret_cast<double2 *>(ut + (size_t)(first + k * kFixWarps) * 60)[lane] = make_double2(u0, u1);
        pa = na;
        pb = nb;
    }
    if (!ok) {
        if (lane == 0) atomicExch(err, 2);
        // drain: wait (bounded) for every copy this warp still has in flight
        for (int c = 0; c < 3; ++c)
            if (c >= chunk || k + 1 < nmine) tc::mbar_wait(&bar[c], (uint32_t)((c >= chunk ? k : k + 1) & 1));
    }
}

// K_e P_e for the k load cases of P (slot-major, P[slot * k + j]) into
// ut[(60 e + i) * k + j]: k_elem_fix with the cases inside the element, so
// that a record is read once for all of them and the products are bitwise
// those of the single-case kernel.  Bound by instruction issue (1.8 ns per
// element and case over the chip, against 6.3 ns by FP64 FMA).
template <bool ROWS>
__global__ void __launch_bounds__(kFixWarps * 32, 1)
k_mr_elem_fix(int nels, int nk, const unsigned char *__restrict__ rec, const int *__restrict__ conn,
              const double *__restrict__ P, double *__restrict__ ut, int *__restrict__ err, const double *__restrict__ km)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned char *stage = smem + (size_t)w * 3 * fx::kChunk0;
    int4 *pq = reinterpret_cast<int4 *>(smem + (size_t)kFixWarps * 3 * fx::kChunk0) + w * 60;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + (size_t)kFixWarps * (3 * fx::kChunk0 + 960)) + 3 * w;
    const int per_cta = (nels + gridDim.x - 1) / gridDim.x;
    const int first = blockIdx.x * per_cta + w, e1 = min(nels, (int)(blockIdx.x + 1) * per_cta);
    if (first >= e1) return;
    if (lane == 0) {
        for (int c = 0; c < 3; ++c) tc::mbar_init(&bar[c], 1);
        tc::mbar_fence_init();
    }
    __syncwarp();
    const uint64_t pol = tc::l2_evict_first_policy();
    auto issue = [&](int c, int e) {
        tc::mbar_expect_tx(&bar[c], fx::chunk_bytes(c));
        tc::bulk_g2s_hint(stage + c * fx::kChunk0, rec + (size_t)e * fx::kRecBytes + fx::chunk_off(c), fx::chunk_bytes(c),
                          &bar[c], pol);
    };
    if (lane == 0)
        for (int c = 0; c < 3; ++c) issue(c, first);
    const int l = lane < 30 ? lane : 29;
    bool ok = true;
    uint32_t parity = 0;
    int e = first, chunk = 0, j = 0;
    for (; e < e1 && ok; e += kFixWarps, parity ^= 1) {
        const int nd = lane < 20 ? conn[(size_t)e * 20 + lane] : 0;
        const int n0 = __shfl_sync(FULLMASK, nd, 2 * l / 3), n1 = __shfl_sync(FULLMASK, nd, (2 * l + 1) / 3);
        const double *qa = P + ((size_t)3 * n0 + 2 * l % 3) * nk, *qb = P + ((size_t)3 * n1 + (2 * l + 1) % 3) * nk;
        double pa = qa[0], pb = qb[0];
        double *o = ut + ((size_t)e * 60 + 2 * l) * nk;
        for (j = 0; j < nk; ++j) {
            const int jn = j + 1 < nk ? j + 1 : j;
            const double na = qa[jn], nb = qb[jn];   // of the next case
            double u0, u1;
            bool weak0, weak1;
            ok = fx::product<ROWS>(
                lane, pa, pb, pq,
                [&](int c) -> const unsigned char * {
                    if (j > 0) return stage + c * fx::kChunk0;
                    chunk = c;
                    return __all_sync(FULLMASK, tc::mbar_wait(&bar[c], parity)) ? stage + c * fx::kChunk0 : nullptr;
                },
                [&](int c) {
                    if (j + 1 < nk) return;
                    __syncwarp();   // every lane is done with the stage
                    if (lane == 0 && e + kFixWarps < e1) {
                        tc::fence_proxy_async();
                        issue(c, e + kFixWarps);
                    }
                },
                u0, u1, weak0, weak1);
            if (!ok) break;
            if (ROWS) fx::weak_rows(lane, pa, pb, km + (size_t)e * 3600, weak0, weak1, u0, u1);
            if (lane < 30) {
                o[j] = u0;
                o[nk + j] = u1;
            }
            pa = na;
            pb = nb;
        }
        if (!ok) break;
    }
    if (!ok) {   // in the first case of element e: chunks from `chunk` on are in flight
        if (lane == 0) atomicExch(err, 2);
        for (int c = chunk; c < 3; ++c) tc::mbar_wait(&bar[c], parity);
    }
}

// The same with one record for every element (PCG_KM), held in shared
// memory; bitwise the products of k_elem_fix on copies of it.  Bound by
// instruction issue: 0.93 ms on an 80^3 cube, k_elem_shared64 3.29 ms.
constexpr int kSharedFixWarps = 8;
template <bool ROWS>
__global__ void __launch_bounds__(kSharedFixWarps * 32, 2)
k_elem_shared_fix(int nels, const unsigned char *__restrict__ rec, const int *__restrict__ conn,
                  const double *__restrict__ p, double *__restrict__ ut, const PcgState *__restrict__ st,
                  const double *__restrict__ km)
{
    __shared__ int4 pq[kSharedFixWarps][60];
    __shared__ __align__(16) unsigned char r[fx::kRecBytes];
    pdl_enter();
    if (st && st->stop) return;
    for (int i = threadIdx.x; i < fx::kRecBytes / 16; i += blockDim.x)
        reinterpret_cast<int4 *>(r)[i] = reinterpret_cast<const int4 *>(rec)[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, stride = gridDim.x * kSharedFixWarps;
    int e = blockIdx.x * kSharedFixWarps + w;
    auto node = [&](int x) { return lane < 20 && x < nels ? conn[(size_t)x * 20 + lane] : 0; };
    int nd = node(e);
    double pa, pb;
    fx::gather2<true>(nd, lane, p, pa, pb);
    nd = node(e + stride);
    for (; e < nels; e += stride) {
        double na, nb, u0, u1;
        bool weak0, weak1;
        fx::gather2<true>(nd, lane, p, na, nb);
        nd = node(e + 2 * stride);
        fx::product<ROWS>(
            lane, pa, pb, pq[w], [&](int c) -> const unsigned char * { return r + fx::chunk_off(c); }, [](int) {}, u0, u1,
            weak0, weak1);
        if (ROWS) fx::weak_rows(lane, pa, pb, km, weak0, weak1, u0, u1);
        if (lane < 30) reinterpret_cast<double2 *>(ut + (size_t)e * 60)[lane] = make_double2(u0, u1);
        pa = na;
        pb = nb;
    }
}

static int fix_launched(Ctx &c, const char *name)
{
    c.launches++;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s: launch failed: %s", name, cudaGetErrorString(e));
        return 1;
    }
    return 0;
}

int launch_pack_storkm(Ctx &c, int nels, const double *km, float *kp, unsigned char *rec, int *bad)
{
    const int grid = nels < c.nsm * 6 ? nels : c.nsm * 6;
    k_pack_storkm<<<grid, kPackThreads, 0, c.stream>>>(nels, km, kp, rec, bad);
    return fix_launched(c, "k_pack_storkm");
}

// Shared-memory attributes of the bulk-copy kernels, set once per context by
// their first products, which are outside any stream capture.
static int fix_attributes(Ctx &c)
{
    if (c.fix_attr) return 0;
    const void *fn[] = {(const void *)k_elem_fix<false>, (const void *)k_elem_fix<true>, (const void *)k_mr_elem_fix<false>,
                        (const void *)k_mr_elem_fix<true>};
    cudaError_t e = cudaSuccess;
    for (const void *f : fn)
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFixSmem);
    if (e != cudaSuccess) {
        set_error("fixed-point products: cannot reserve %zu bytes of shared memory: %s", kFixSmem, cudaGetErrorString(e));
        return 1;
    }
    c.fix_attr = true;
    return 0;
}

int launch_elem_fix(Ctx &c, const double *p, const PcgState *st, bool rows)
{
    if (fix_attributes(c)) return 1;
    // one CTA per SM, and on small meshes as few warps per SM as the mesh has
    const int grid = c.nels < c.nsm ? c.nels : c.nsm;
    launch_dependent(c.dependent && st, c.stream, grid, kFixWarps * 32, kFixSmem,
                     rows ? k_elem_fix<true> : k_elem_fix<false>, c.nels, c.kmfix, c.conn, p, (double *)c.utemp, st, c.kerr,
                     c.km64);
    return fix_launched(c, "k_elem_fix");
}

int launch_mr_elem_fix(Ctx &c, int k, const double *P, double *ut, bool rows)
{
    if (fix_attributes(c)) return 1;
    const int grid = c.nels < c.nsm ? c.nels : c.nsm;
    auto kernel = rows ? k_mr_elem_fix<true> : k_mr_elem_fix<false>;
    kernel<<<grid, kFixWarps * 32, kFixSmem, c.stream>>>(c.nels, k, c.kmfix, c.conn, P, ut, c.kerr, c.km64);
    return fix_launched(c, "k_mr_elem_fix");
}

int launch_elem_shared_fix(Ctx &c, const double *p, const PcgState *st, bool rows)
{
    const int nb = (c.nels + kSharedFixWarps - 1) / kSharedFixWarps;
    const int grid = nb < c.nsm * 2 ? nb : c.nsm * 2;
    launch_dependent(c.dependent && st, c.stream, grid, kSharedFixWarps * 32, 0,
                     rows ? k_elem_shared_fix<true> : k_elem_shared_fix<false>, c.nels, c.skmfix, c.conn, p, (double *)c.utemp, st,
                     c.skm64);
    return fix_launched(c, "k_elem_shared_fix");
}

}  // namespace pf
