// pf_fix.cuh -- FP64-class element products in 64-bit fixed point.
//
// GB300 runs two FP64 FMA per SM and clock but sixty-four 32 x 32 -> 64 bit
// integer multiply-adds, so the 3,600 FP64 FMA of K_e p_e (1,800 clocks of an
// SM per element) are formed in integers instead.  A symmetric K_e is scaled
// to K'(i,j) = K(i,j) 2^(s_i + s_j) with every K'(i,i) in [1/4, 1) and held
// as integers of 57 bits below the point, each entry once (30 cyclic 2 x 2
// block diagonals): 14.8 KB per element instead of 28.8.  p_e becomes
// p_j 2^(-s_j), scaled by the element's largest, in 57 bits too.  Both are
// split into a high word and a signed 29-bit low word; three of the four
// cross products are summed EXACTLY (no carry can leave 63 bits:
// 60 x 2^28 x 2^28 and 60 x 2 x 2^56), so a result does not depend on the
// order of its terms and is rounded once, when it becomes FP64 again.
//
// Dropped are bits of K' and p' below 2^-57 and the product of the two low
// words: per row at most 60 x 3 x 2^-58 in the scaled units, that is
//     |error of u_i| <= 2^-47 sqrt(K_ii) max_j sqrt(K_jj) |p_j|,
// a bound by the element's largest scaled value, not by the row's own terms.
// In the 2-norm of D^(-1/2) u (D the diagonal) the error is a fifth to two
// fifths of that of 60 FP64 FMA, also in thin and distorted elements, whose
// rows differ in size; that is the norm in which a Jacobi-scaled PCG sees
// it, so the solves and their true residuals take this product.  A row
// whose terms K_ij p_j are all small beside the element's largest scaled
// value has fewer correct bits than by FMA, none at 2^-57 of it; the
// products that a caller asks for (pf_ebe_matvec) form such rows again by
// FMA (weak_rows).
#pragma once
#include "pf_device.cuh"

namespace pf {
namespace fx {

constexpr int kLow = 29;                    // bits of the low word
constexpr int kNoKey = -(1 << 28);          // exponent of a zero

// One element's record: three chunks, each one copy into shared memory.
// Block diagonal s = 1..14 holds block (l, l+s) of the 30 block rows l as
// two rows of 30 x 16 bytes (entries (0,0), (0,1), then (1,0), (1,1), each a
// high and a low word), diagonal 15 its 15 blocks likewise, diagonal 0 the
// entries (0,0), (0,1) and apart from them (1,1).
//   chunk 0: s_i and the extra bits, diagonals 0, 15, 14, 13, 12, 11
//   chunk 1: diagonals 10 .. 6        chunk 2: diagonals 5 .. 1
constexpr int kOffExp = 0;                  // s_i, 60 16-bit integers
constexpr int kOffExtra = 120;              // bits below 2^-57 that the entries have (0 or 2), a 16-bit integer
constexpr int kOff0 = 128;
constexpr int kOff11 = kOff0 + 480;
constexpr int kOff15 = kOff11 + 240;
constexpr int kChunk0 = kOff15 + 480 + 4 * 960 + 16;   // a multiple of 32, as every offset of a chunk
constexpr int kChunk = 5 * 960;
constexpr int kRecBytes = kChunk0 + 2 * kChunk;
static_assert(kChunk0 % 32 == 0 && kChunk % 32 == 0, "chunks are whole sectors");
__host__ __device__ __forceinline__ constexpr int chunk_off(int c) { return c == 0 ? 0 : kChunk0 + (c - 1) * kChunk; }
__host__ __device__ __forceinline__ constexpr int chunk_bytes(int c) { return c == 0 ? kChunk0 : kChunk; }
// byte offset in its chunk of row h of block diagonal s = 1..15
__host__ __device__ __forceinline__ constexpr int row_off(int s, int h)
{
    return s == 15 ? kOff15 + 240 * h : s > 10 ? kOff15 + 480 + 960 * (14 - s) + 480 * h : 960 * ((10 - s) % 5) + 480 * h;
}

// magnitude and exponent of a double: |x| = m 2^(ex - 1075)
__host__ __device__ __forceinline__ long long bits_mant(long long b, int &ex)
{
    const int e = (int)((b >> 52) & 0x7ff);
    ex = e ? e : 1;
    return (b & ((1LL << 52) - 1)) | (e ? 1LL << 52 : 0);
}

// m 2^(4 - sh), rounded to nearest (m < 2^53, sh >= 0): below 2^57
__host__ __device__ __forceinline__ long long shift_round(long long m, int sh)
{
    const int n = sh < 62 ? sh : 62;
    return ((m << 4) + ((1LL << n) >> 1)) >> n;
}

struct Words {
    int h, l;   // value = h 2^29 + l, -2^28 <= l < 2^28
};

__host__ __device__ __forceinline__ Words split(long long v)
{
    Words w;
    w.l = (int)((long long)((unsigned long long)v << (64 - kLow)) >> (64 - kLow));
    w.h = (int)((v - w.l) >> kLow);
    return w;
}

// K(i,k) 2^(s_i + s_k) in 57 + extra fractional bits; false when it is not
// below 1 in magnitude (not a positive semi-definite matrix) or not finite
__host__ __device__ __forceinline__ bool fix_entry(long long kbits, int si, int sk, int extra, Words &w)
{
    int ex;
    const long long m = bits_mant(kbits, ex) << extra;   // below 2^55
    const int sh = 1022 - ex - si - sk;
    const bool ok = (sh >= 0 && ex < 2047) || m == 0;
    const long long v = ok ? shift_round(m, m == 0 ? 62 : sh) : 0;
    w = split(kbits < 0 ? -v : v);
    return ok;
}

// |K(i,k)| 2^(s_i + s_k) in 20 fractional bits, rounded up
__host__ __device__ __forceinline__ int fix_size(long long kbits, int si, int sk)
{
    int ex;
    const long long m = bits_mant(kbits, ex);
    const int sh = 1022 - ex - si - sk;
    return m == 0 || sh >= 30 ? 1 : (int)(m >> 33 >> (sh < 0 ? 0 : sh)) + 1;
}

// s_i of a diagonal entry K(i,i) = f 2^e, f in [1/2, 1): K(i,i) 4^s in [1/4, 1)
__host__ __device__ __forceinline__ int fix_scale(long long kbits)
{
    const int e = (int)((kbits >> 52) & 0x7ff) - 1022;
    return -((e + 4096 + 1) / 2 - 2048);   // -ceil(e / 2)
}

// (long long)a * b + c (written so in C: 1.61 instead of 1.41 ms of an 80^3 product)
__device__ __forceinline__ long long madw(int a, int b, long long c)
{
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}

struct Sums {
    long long h0 = 0, m0 = 0, h1 = 0, m1 = 0;   // high x high, and the two mixed products, of two rows
};

// rows (a, b) of a 2 x 2 block times the two values of q = (h, l, h, l)
__device__ __forceinline__ void block_fwd(Sums &s, const int4 a, const int4 b, const int4 q)
{
    s.h0 = madw(a.x, q.x, s.h0);
    s.h1 = madw(b.x, q.x, s.h1);
    s.m0 = madw(a.x, q.y, s.m0);
    s.m1 = madw(b.x, q.y, s.m1);
    s.m0 = madw(a.y, q.x, s.m0);
    s.m1 = madw(b.y, q.x, s.m1);
    s.h0 = madw(a.z, q.z, s.h0);
    s.h1 = madw(b.z, q.z, s.h1);
    s.m0 = madw(a.z, q.w, s.m0);
    s.m1 = madw(b.z, q.w, s.m1);
    s.m0 = madw(a.w, q.z, s.m0);
    s.m1 = madw(b.w, q.z, s.m1);
}
// and its transpose
__device__ __forceinline__ void block_bwd(Sums &s, const int4 a, const int4 b, const int4 q)
{
    block_fwd(s, make_int4(a.x, a.y, b.x, b.y), make_int4(a.z, a.w, b.z, b.w), q);
}

// The largest |K'(i,j) p'(j)| of two rows in 28 + extra fractional bits, from
// the high words, for weak_rows
struct Largest {
    unsigned a = 0, b = 0;
};
__device__ __forceinline__ void larger_fwd(Largest &s, const int4 a, const int4 b, const int4 q)
{
    const unsigned q0 = (unsigned)abs(q.x) << 3, q1 = (unsigned)abs(q.z) << 3;
    s.a = max(s.a, max(__umulhi((unsigned)abs(a.x) << 1, q0), __umulhi((unsigned)abs(a.z) << 1, q1)));
    s.b = max(s.b, max(__umulhi((unsigned)abs(b.x) << 1, q0), __umulhi((unsigned)abs(b.z) << 1, q1)));
}
__device__ __forceinline__ void larger_bwd(Largest &s, const int4 a, const int4 b, const int4 q)
{
    larger_fwd(s, make_int4(a.x, a.y, b.x, b.y), make_int4(a.z, a.w, b.z, b.w), q);
}
constexpr int kWeakBits = 5;   // a row whose terms are all below 2^-5 of the scaled units is a weak one

__device__ __forceinline__ Sums shift_from(const Sums &s, int src)
{
    Sums t;
    t.h0 = __shfl_sync(FULLMASK, s.h0, src);
    t.m0 = __shfl_sync(FULLMASK, s.m0, src);
    t.h1 = __shfl_sync(FULLMASK, s.h1, src);
    t.m1 = __shfl_sync(FULLMASK, s.m1, src);
    return t;
}

// A value of p as the element's fixed point sees it: bits, and the exponent
// key of p 2^(-s) (kNoKey for zero)
__device__ __forceinline__ int fix_key(long long b, int s)
{
    int ex;
    const long long m = bits_mant(b, ex);
    return m ? ex - s : kNoKey;
}
__device__ __forceinline__ Words fix_value(long long b, int key, int kmax)
{
    int ex;
    const long long m = bits_mant(b, ex);
    const long long v = key == kNoKey ? 0 : shift_round(m, kmax - key);
    return split(b < 0 ? -v : v);
}

// h 2^58 + m 2^29 (units of 2^-114 of the scaled product, less the extra
// bits) back to the row's scale: kmax is the largest exponent key of p, s
// the row's exponent.  The sum is regrouped into two parts that are exact as
// doubles, so it is rounded once.
__device__ __forceinline__ double fix_result(long long h, long long m, int kmax, int s)
{
    h += m >> kLow;
    const long long low = (h & ((1LL << 22) - 1)) << kLow | (m & ((1LL << kLow) - 1));   // 51 bits
    const double v = fma((double)(h >> 22), 2251799813685248.0, (double)low);
    int t = kmax - s - (1022 + 114 - kLow);
    t = t < -2040 ? -2040 : (t > 2040 ? 2040 : t);
    const int t1 = t / 2, t2 = t - t1;
    return v * __longlong_as_double((long long)(t1 + 1023) << 52) * __longlong_as_double((long long)(t2 + 1023) << 52);
}

// Products of one element by one warp.  Lane l < 30 owns rows and values 2l
// and 2l + 1 (lanes 30 and 31 repeat lane 29).  Block (l, l+s) serves two
// rows of lane l, and by symmetry two rows of lane l + s: those sums are
// handed to the next lane as s goes down from 15, so that lane l always
// holds the sums of lane l + s and each lane receives its own at the end.
// Every entry is loaded once and multiplied twelve times.  pq: 60 int4 of
// shared memory per warp, the words of p twice over so that l + s needs no
// wrap.  Chunk c of the record is read between enter(c), which returns its
// address or null to give up (product() then returns false), and leave(c).
// ROWS: weak0 and weak1 say which of the two rows weak_rows has to form.
template <bool ROWS, typename Enter, typename Leave>
__device__ __forceinline__ bool product(int lane, double pa, double pb, int4 *__restrict__ pq, Enter enter, Leave leave,
                                        double &u0, double &u1, bool &weak0, bool &weak1)
{
    const int l = lane < 30 ? lane : 29, prev = lane == 0 ? 29 : l - 1;
    const unsigned char *r = enter(0);
    if (!r) return false;
    const short2 ex = *reinterpret_cast<const short2 *>(r + kOffExp + 4 * l);
    const int extra = *reinterpret_cast<const short *>(r + kOffExtra);
    const long long ba = __double_as_longlong(pa), bb = __double_as_longlong(pb);
    const int qa = fix_key(ba, ex.x), qb = fix_key(bb, ex.y);
    const int kmax = __reduce_max_sync(FULLMASK, qa > qb ? qa : qb);
    const bool finite = !__any_sync(FULLMASK, ((ba >> 52) & 0x7ff) == 0x7ff || ((bb >> 52) & 0x7ff) == 0x7ff);
    const Words wa = fix_value(ba, qa, kmax), wb = fix_value(bb, qb, kmax);
    const int4 own = make_int4(wa.h, wa.l, wb.h, wb.l);
    if (lane < 30) {
        pq[lane] = own;
        pq[lane + 30] = own;
    }
    __syncwarp();
    Sums f, t;
    Largest lf, lt;
    {
        const int4 k0 = *reinterpret_cast<const int4 *>(r + kOff0 + 16 * l);
        const int2 k11 = *reinterpret_cast<const int2 *>(r + kOff11 + 8 * l);
        block_fwd(f, k0, make_int4(k0.z, k0.w, k11.x, k11.y), own);
        if constexpr (ROWS) larger_fwd(lf, k0, make_int4(k0.z, k0.w, k11.x, k11.y), own);
    }
    {
        const int l15 = l < 15 ? l : 14;
        int4 a = *reinterpret_cast<const int4 *>(r + row_off(15, 0) + 16 * l15);
        int4 b = *reinterpret_cast<const int4 *>(r + row_off(15, 1) + 16 * l15);
        if (l >= 15) a = b = make_int4(0, 0, 0, 0);
        block_fwd(f, a, b, pq[l + 15]);
        block_bwd(t, a, b, own);
        if constexpr (ROWS) {
            larger_fwd(lf, a, b, pq[l + 15]);
            larger_bwd(lt, a, b, own);
        }
    }
    const int4 *pl = pq + l;
    auto diagonal = [&](const unsigned char *rl, int s) {   // rl: the chunk, at this lane's 16 bytes
        const int4 a = *reinterpret_cast<const int4 *>(rl + row_off(s, 0));
        const int4 b = *reinterpret_cast<const int4 *>(rl + row_off(s, 1));
        t = shift_from(t, prev);
        block_fwd(f, a, b, pl[s]);
        block_bwd(t, a, b, own);
        if constexpr (ROWS) {
            lt.a = __shfl_sync(FULLMASK, lt.a, prev);
            lt.b = __shfl_sync(FULLMASK, lt.b, prev);
            larger_fwd(lf, a, b, pl[s]);
            larger_bwd(lt, a, b, own);
        }
    };
    r += 16 * l;
#pragma unroll
    for (int s = 14; s >= 11; --s) diagonal(r, s);
    leave(0);
#pragma unroll 1
    for (int c = 1; c < 3; ++c) {
        r = enter(c);
        if (!r) return false;
        r += 16 * l;
#pragma unroll
        for (int s = 10; s >= 6; --s) diagonal(r, s);   // diagonals 5..1 lie as 10..6 do
        pl -= 5;
        leave(c);
    }
    t = shift_from(t, prev);
    __syncwarp();   // pq is free again
    u0 = fix_result(f.h0 + t.h0, f.m0 + t.m0, kmax - extra, ex.x);
    u1 = fix_result(f.h1 + t.h1, f.m1 + t.m1, kmax - extra, ex.y);
    if (!finite) u0 = u1 = __longlong_as_double(0x7ff8000000000000LL);
    if constexpr (ROWS) {
        const unsigned bound = 1u << (28 + extra - kWeakBits);
        const bool any = kmax != kNoKey;   // p_e = 0: so is the product
        weak0 = !finite || (max(lf.a, __shfl_sync(FULLMASK, lt.a, prev)) < bound && any);
        weak1 = !finite || (max(lf.b, __shfl_sync(FULLMASK, lt.b, prev)) < bound && any);
    }
    return true;
}
template <typename Enter, typename Leave>
__device__ __forceinline__ bool product(int lane, double pa, double pb, int4 *__restrict__ pq, Enter enter, Leave leave,
                                        double &u0, double &u1)
{
    bool weak0, weak1;
    return product<false>(lane, pa, pb, pq, enter, leave, u0, u1, weak0, weak1);
}

// The weak rows of an element by FMA, in k_elem's order, from its matrix ke.
// Largest error of a row over the sum of its |K_ij p_j|, and the 2-norm of
// all errors over 2^-53 that of the sums, 40 bricks of 100 x 1 x 0.02:
//                             fixed point      FMA            with this
//   normal p                  2^-52.6  0.27    2^-51.3  0.59  2^-52.6  0.27
//   one p = 1, rest 1e-9      2^-34.7  0.53    2^-50.1  1.94  2^-50.1  0.44
//   p over 20 decades         2^-43.3  0.46    2^-50.5  0.84  2^-50.5  0.45
__device__ __forceinline__ void weak_rows(int lane, double pa, double pb, const double *__restrict__ ke, bool weak0, bool weak1,
                                          double &u0, double &u1)
{
    if (!__any_sync(FULLMASK, weak0 || weak1)) return;
    const double *kr = ke + 2 * (lane < 30 ? lane : 29);
    double a0 = 0.0, a1 = 0.0;
#pragma unroll 6
    for (int j = 0; j < 60; j += 2) {
        const double p0 = __shfl_sync(FULLMASK, pa, j >> 1), p1 = __shfl_sync(FULLMASK, pb, j >> 1);
        const double2 k0 = __ldg(reinterpret_cast<const double2 *>(kr + 60 * j));
        const double2 k1 = __ldg(reinterpret_cast<const double2 *>(kr + 60 * j + 60));
        a0 = fma(k0.x, p0, a0);
        a1 = fma(k0.y, p0, a1);
        a0 = fma(k1.x, p1, a0);
        a1 = fma(k1.y, p1, a1);
    }
    if (weak0) u0 = a0;
    if (weak1) u1 = a1;
}

// Lane l's part of the connectivity is node l; p at its two freedoms.  NC: p
// was written by an earlier launch.
template <bool NC>
__device__ __forceinline__ void gather2(int nd, int lane, const double *__restrict__ p, double &pa, double &pb)
{
    const int l = lane < 30 ? lane : 29, j0 = 2 * l, j1 = 2 * l + 1;
    const int n0 = __shfl_sync(FULLMASK, nd, j0 / 3), n1 = __shfl_sync(FULLMASK, nd, j1 / 3);
    const double *qa = p + (size_t)3 * n0 + j0 % 3, *qb = p + (size_t)3 * n1 + j1 % 3;
    pa = NC ? __ldg(qa) : __ldcg(qa);
    pb = NC ? __ldg(qb) : __ldcg(qb);
}

// u_e = K_e p_e of element e from its record where it lies, into ut[60 e]:
// the same sums as k_elem_fix's, so bitwise its results
template <bool NC>
__device__ __forceinline__ void elem_warp(size_t e, int lane, const unsigned char *__restrict__ rec,
                                          const int *__restrict__ conn, const double *__restrict__ p,
                                          double *__restrict__ ut, int4 *__restrict__ pq)
{
    const int nd = lane < 20 ? conn[e * 20 + lane] : 0;
    double pa, pb, u0, u1;
    gather2<NC>(nd, lane, p, pa, pb);
    product(
        lane, pa, pb, pq, [&](int c) { return rec + e * kRecBytes + chunk_off(c); }, [](int) {}, u0, u1);
    if (lane < 30) reinterpret_cast<double2 *>(ut + e * 60)[lane] = make_double2(u0, u1);
}

}  // namespace fx
}  // namespace pf
