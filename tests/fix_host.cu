// The fixed-point record's helpers as the library's kernels use them
// (pf_fix.cuh), compiled for the host: entry points for test_fixed_point.py.
#include "pf_fix.cuh"

#include <cstring>

namespace fx = pf::fx;

static long long bits(double x)
{
    long long b;
    memcpy(&b, &x, sizeof b);
    return b;
}

extern "C" int fix_scale(double k) { return fx::fix_scale(bits(k)); }
extern "C" int fix_size(double k, int si, int sk) { return fx::fix_size(bits(k), si, sk); }
extern "C" int fix_entry(double k, int si, int sk, int extra, int *h, int *l)
{
    fx::Words w;
    const bool ok = fx::fix_entry(bits(k), si, sk, extra, w);
    *h = w.h;
    *l = w.l;
    return ok;
}
extern "C" int row_off(int s, int h) { return (s > 10 ? 0 : s > 5 ? fx::chunk_off(1) : fx::chunk_off(2)) + fx::row_off(s, h); }
extern "C" int record_bytes() { return fx::kRecBytes; }
