// The plane-sweep tile engine shared by the single-view kernel (sweep.cu) and the persistent
// batched kernel (batch.cu): warp + windowed ZNCC + best-k over sources + streaming
// winner-take-all for one TW x TH output tile and one contiguous range of hypotheses.
//
// Semantics follow the reference's fused CPU step (_dense.pyx:740-838 with _sweep.h) and its
// definitional form (_dense.ncc_warp + _dense.combine, _dense.pyx:13-144):
//   * a source sample is valid when its camera-frame Z > 1e-6, 0 <= u <= w - 1.001,
//     0 <= v <= h - 1.001 and the bilinear value is finite (NaN pixels are masks);
//   * window sums run over the (2r+1)^2 window clipped to the reference image;
//     count/k^2 <= 0.9 gives NCC = -1; otherwise
//     NCC = (mean(JI) - mu mean(J)) / (sd * sdj), sdj = sqrt(var(J)) if var > 1e-6 else 1e-3,
//     clipped to [-1, 1];
//   * the hypothesis score is the float32 mean of the top_k source NCCs (summed in descending
//     order); the winner update is strict '>' in hypothesis order (first index wins ties),
//     tracking the score of the previous hypothesis and of the one after the winner.
//
// Work of one CTA per (hypothesis, source):
//   A. warp the source into a shared-memory tile with an r-pixel halo (NaN = invalid sample);
//   B. horizontal window sums of (V, J, J^2, J*I): each thread runs along a 16-column row
//      segment (inputs from 16-byte shared loads, products formed once per input) and stores
//      one float4 per output;
//   C. vertical running sums down each column (TH/SEG rows per thread) from float4 loads, NCC,
//      insertion into a per-pixel top-k list in registers.
// After the last source the winner-take-all state of each pixel is updated in registers; it
// leaves the SM once per hypothesis chunk. Window sums are short FP32 sums (at most TH/SEG
// add/subtract steps): within the parity bar wherever the window has texture, but on bright
// low-texture windows at r <= 2 their rounding, amplified by 1 / (sd_ref sd_src), can reach
// ~1e-3 in NCC. X64 (MVS_PREC_FP64_SUMS) keeps the sums in float64 as the reference does
// (stage_b64 / stage_c64).
#pragma once

#include "common.cuh"

namespace mvs {

constexpr int TW = 64;                 // output tile width (columns)
constexpr int ROWS = 8;                // output rows per thread in stage C
constexpr int TH_DEFAULT = 32;         // output tile height of the default shape

// A TW x TH output tile runs on NT = 8 TH threads: thread t keeps column t mod TW and the ROWS rows
// of segment t / TW in stage C, so every thread's rows start on a multiple of 8 in each of the
// three shapes (TH = 16, 32, 64; 128, 256, 512 threads).
template <int TH>
struct TileShape {
    static_assert(TH == 16 || TH == 32 || TH == 64, "tile height 16, 32 or 64");
    static constexpr int NT = 8 * TH;              // threads per CTA
    static constexpr int SEG = NT / TW;            // row segments (= TH / ROWS)
    static constexpr int MIN_CTAS = TH == 16 ? 3 : (TH == 32 ? 2 : 1);   // resident CTAs per SM
};

struct SrcGeo {
    const void* img;                   // float or __half, (h, w) row-major
    int h, w;
    double m[9];                       // PLANES: A = Rs R_ref^T K_ref^-1; ray path: Rs
    double b[3];                       // Rs (C_ref - C_src)
    double f, k1, k2, k3, cx, cy;
};

struct SweepParams {
    CUtensorMap ref_map;               // 2D tiled map of `ref` (single-view kernel, ref_tma = 1)
    int ref_tma;                       // 1: the reference tile is copied by TMA
    int H, W, n_src, kk;
    int topk_bottom;                   // 1: keep the n-kk lowest and subtract from the total
    int i0, i1, ppc;                   // hypotheses [i0, i1), planes per chunk
    int hyp_kind, t0;
    int r, nchunks;
    int fresh;                         // 1: start from the initial state instead of loading it
    unsigned wait_limit;               // try_wait iterations of the TMA tile wait
    long long map_stride;
    const float* ref;
    const float* mu;
    const float* sd;
    const float* ray;
    const float* hyp_a;                // MAPS: maps; LINEAR/REFINE: base
    const float* hyp_b;                // LINEAR/REFINE: step
    float* best;
    float* prev;
    float* spb;
    float* snb;
    int* idx;
    float* rec;                        // chunk records (6, nchunks, H, W) or nullptr
    SrcGeo src[MVS_MAX_SOURCES];
    float planes[MVS_MAX_PLANES_PER_CALL];   // PLANES: inverse depth of hypothesis i0 + j
};

// Per (hypothesis, source, tile) projective map in tile-local coordinates (a, b) of the halo
// origin, composed in FP64 and rounded once: u_l = (nu0 + nu1 a + nu2 b) / dz, v_l likewise,
// dz = dz0 + dz1 a + dz2 b; the source pixel is (U0 + u_l, V0 + v_l) and the camera-frame
// depth is zs * dz. Small local magnitudes keep the FP32 evaluation at ~1e-5 px.
// The nine map coefficients are kept twice side by side, as the operands of packed float32 pairs
// (two samples per instruction).
struct Coef {
    float2 nu0, nu1, nu2, nv0, nv1, nv2, dz0, dz1, dz2;
    float zs, lo_u, hi_u, lo_v, hi_v;
    int U0, V0;
    int inside;       // MAP_INSIDE / MAP_OUTSIDE: every sample of the halo rectangle is valid / invalid
};

// Where the halo rectangle of a tile maps to in the source (with a margin of 1e-3 px, which absorbs
// the FP32 evaluation error of ~1e-5 px); MAP_MIXED: each sample is tested.
enum { MAP_MIXED = 0, MAP_INSIDE = 1, MAP_OUTSIDE = 2 };

template <int R, int TH = TH_DEFAULT>
struct Geom {
    static constexpr int K = 2 * R + 1;
    static constexpr int RA = (R + 3) & ~3;        // halo rounded up to a float4
    static constexpr int HR = TH + 2 * R;          // sampled rows
    static constexpr int HC = TW + 2 * R;          // sampled columns
    static constexpr int JP = TW + 2 * RA + 4;     // shared row pitch (floats): odd in float4 units
    static constexpr int P = 16;                   // stage-B outputs per thread (one row segment)
    static constexpr int NSEG = TW / P;
    static constexpr int NIN = P + 2 * RA;         // stage-B inputs per segment
    static constexpr size_t count_bytes() {      // compensated mode: uint8 horizontal window counts
        return ((size_t)HR * TW + 15) & ~(size_t)15;
    }
    static constexpr size_t smem_bytes(int winner_planes = 6) {       // sJ, sI, sH, winner state, sC
        return (size_t)HR * JP * 4 * 2 + (size_t)HR * TW * 16 + (size_t)winner_planes * TH * TW * 4 +
               sizeof(Coef) * MVS_MAX_SOURCES;
    }
};

// Planes of the winner state in shared memory: best, prev, s_prev_best, s_next_best, idx and, unless
// FIRST_TO_REC, a chunk record's first score, which then goes to the record when it is formed. At
// R = 4 and 5 leaving that plane out lets two CTAs share an SM (1003 x 749, R = 5, float64 sums: 8.0
// -> 6.7 ms); elsewhere it changes no occupancy, and the store inside the loop costs registers
// (R = 3: 101.9 -> 114.6 ms).
template <int R, int KMAX, int TH>
struct WinnerState {
    static constexpr bool FIRST_TO_REC = TH == TH_DEFAULT && KMAX == 2 && (R == 4 || R == 5);
    static constexpr int PLANES = FIRST_TO_REC ? 5 : 6;
};

// Largest shared-memory footprint over radii 0..RMAX (a persistent CTA serves any of them).
template <int RMAX, int TH = TH_DEFAULT>
constexpr size_t smem_bytes_upto() {
    size_t m = 0;
    if constexpr (RMAX >= 0) m = Geom<0, TH>::smem_bytes() > m ? Geom<0, TH>::smem_bytes() : m;
    if constexpr (RMAX >= 1) m = Geom<1, TH>::smem_bytes() > m ? Geom<1, TH>::smem_bytes() : m;
    if constexpr (RMAX >= 2) m = Geom<2, TH>::smem_bytes() > m ? Geom<2, TH>::smem_bytes() : m;
    if constexpr (RMAX >= 3) m = Geom<3, TH>::smem_bytes() > m ? Geom<3, TH>::smem_bytes() : m;
    if constexpr (RMAX >= 4) m = Geom<4, TH>::smem_bytes() > m ? Geom<4, TH>::smem_bytes() : m;
    if constexpr (RMAX >= 5) m = Geom<5, TH>::smem_bytes() > m ? Geom<5, TH>::smem_bytes() : m;
    if constexpr (RMAX >= 6) m = Geom<6, TH>::smem_bytes() > m ? Geom<6, TH>::smem_bytes() : m;
    if constexpr (RMAX >= 7) m = Geom<7, TH>::smem_bytes() > m ? Geom<7, TH>::smem_bytes() : m;
    return m;
}

__device__ __forceinline__ float qnan() { return __int_as_float(0x7fc00000); }

// Position of the horizontal-sum float4 of (row, col) in shared memory: an XOR swizzle of the
// column's low 3 bits by (segment + row), so that the row-segment writers of stage B (32 lanes =
// 8 rows x 4 segments) and the column readers of stage C (32 consecutive columns) both touch 8
// distinct 16-byte bank groups per quarter-warp.
__device__ __forceinline__ int hs_index(int row, int col) {
    return row * TW + (col ^ (((col >> 4) + row) & 7));
}

__device__ __forceinline__ float hyp_value(const SweepParams& p, int i, int gx, int gy) {
    const long long o = (long long)gy * p.W + gx;
    switch (p.hyp_kind) {
        case MVS_HYP_MAPS:
            return __ldg(p.hyp_a + (long long)(i - p.i0) * p.map_stride + o);
        case MVS_HYP_LINEAR: {      // (base + (float)i * step), two float32 roundings
            const float t = __fmul_rn((float)i, __ldg(p.hyp_b + o));
            return __fadd_rn(__ldg(p.hyp_a + o), t);
        }
        case MVS_HYP_REFINE: {      // max(iu + (float)t * ds, 1e-6), NaN propagating
            const float t = __fmul_rn((float)(i + p.t0), __ldg(p.hyp_b + o));
            return max_nan(__fadd_rn(__ldg(p.hyp_a + o), t), 1e-6f);
        }
        default:
            return p.planes[i - p.i0];
    }
}

template <bool F16>
__device__ __forceinline__ float tap(const void* img, long long i) {
    if constexpr (F16) {
        return __half2float(__ldg(reinterpret_cast<const __half*>(img) + i));
    } else {
        return __ldg(reinterpret_cast<const float*>(img) + i);
    }
}

__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }
// a - b elementwise, one rounding (x (-1) + y is exact before it)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, dup2(-1.0f), a); }
// The hardware's approximations for normal arguments (subnormals flush): the bits of
// __fdividef(1, x) and rsqrtf(x) there, without the steps that scale subnormal arguments.
__device__ __forceinline__ float rcp_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// Finite: stage A leaves NaN at invalid samples, and the value itself where a non-finite source
// pixel entered it.
__device__ __forceinline__ bool finite_value(float x) { return fabsf(x) <= 3.402823466e38f; }
// NCC clipped to [-1, 1], NaN staying NaN
__device__ __forceinline__ float clip_ncc(float x) {
    asm("min.NaN.f32 %0, %0, 0f3F800000;" : "+f"(x));
    asm("max.NaN.f32 %0, %0, 0fBF800000;" : "+f"(x));
    return x;
}

// floor(x) for |x| < 2^22 on the FMA pipe: adding 1.5 * 2^23 rounded toward -inf leaves floor(x)
// in the low mantissa bits. Returns the integer; `f` receives floor(x) as a float.
__device__ __forceinline__ int floor_fma(float x, float& f) {
    const float t = __fadd_rd(x, 12582912.0f);
    f = __fsub_rn(t, 12582912.0f);
    return __float_as_int(t) - 0x4B400000;
}

// Homography path sample (pinhole, constant inverse depth per hypothesis), branch-free so that
// the loads of several samples can be in flight together. Invalid samples read a safe address
// and return NaN.
template <bool F16>
__device__ __forceinline__ float sample_plane(const Coef& c, const void* img, int w, int h, float a, float b, bool in) {
    const float dz = fmaf(c.dz1.x, a, fmaf(c.dz2.x, b, c.dz0.x));
    const float rz = __fdividef(1.0f, dz);
    const float ul = fmaf(c.nu1.x, a, fmaf(c.nu2.x, b, c.nu0.x)) * rz;
    const float vl = fmaf(c.nv1.x, a, fmaf(c.nv2.x, b, c.nv0.x)) * rz;
    bool ok = in && (c.zs * dz > 1e-6f) && (ul >= c.lo_u) && (ul <= c.hi_u) && (vl >= c.lo_v) && (vl <= c.hi_v);
    float fu, fv;
    const int x0 = c.U0 + floor_fma(ok ? ul : 0.f, fu);
    const int y0 = c.V0 + floor_fma(ok ? vl : 0.f, fv);
    // integer guard: every tap stays inside the image whatever the float rounding did
    ok = ok && (unsigned)x0 < (unsigned)(w - 1) && (unsigned)y0 < (unsigned)(h - 1);
    const long long o = ok ? (long long)y0 * w + x0 : 0;
    MVS_BOUND(o >= 0 && o + w + 1 < (long long)h * w);
    const float fx = ul - fu, fy = vl - fv;
    const float a00 = tap<F16>(img, o), a01 = tap<F16>(img, o + 1);
    const float a10 = tap<F16>(img, o + w), a11 = tap<F16>(img, o + w + 1);
    const float top = fmaf(fx, a01 - a00, a00);
    const float bot = fmaf(fx, a11 - a10, a10);
    const float val = fmaf(fy, bot - top, top);
    return (ok && isfinite(val)) ? val : qnan();
}

// Homography samples when the whole halo rectangle is known to map inside the source and to lie
// inside the reference image: no per-sample bounds, two samples at (a.x, b.x) and (a.y, b.y) in
// packed float32 arithmetic (each element rounds as its scalar operation). The FMA pipe runs
// packed pairs at the scalar rate (measured: 126 against 124 FMA a clock per SM), but a pair takes
// one issue slot, and issue is what bounds the kernel: with stage C's packed sums and the
// approximations without subnormal steps, 4000 x 3000, 8 sources, 256 planes 98.8 -> 92.4 ms,
// batch of 8 uneven FP16 views 106.3 -> 99.7 ms. A non-finite source pixel gives a non-finite value,
// which stages B count as invalid.
// `img` / `img1`: the source and its second row; ub, vb: the anchor (U0, V0) less the floor's bias.
// (Evaluating the maps column part first, so that a thread walking down one halo column keeps
// fmaf(x1, a, x0), and clamping the linear tap offset once instead of each coordinate measured
// 1.3 % slower at C2: 167.5 vs 165.2 ms.)
template <bool F16>
__device__ __forceinline__ float2 sample_plane_inside2(const Coef& c, const void* img, const void* img1, int w, int h,
                                                       int ub, int vb, float2 a, float2 b) {
    const float2 bias = dup2(12582912.0f), nbias = dup2(-12582912.0f);
    const float2 dz = __ffma2_rn(c.dz1, a, __ffma2_rn(c.dz2, b, c.dz0));
    const float2 rz = make_float2(rcp_ftz(dz.x), rcp_ftz(dz.y));
    const float2 ul = __fmul2_rn(__ffma2_rn(c.nu1, a, __ffma2_rn(c.nu2, b, c.nu0)), rz);
    const float2 vl = __fmul2_rn(__ffma2_rn(c.nv1, a, __ffma2_rn(c.nv2, b, c.nv0)), rz);
    // floor as floor_fma; the clamp is a no-op when the corner test holds; it keeps every tap inside
    // the image even if an extreme geometry defeated that test
    const float2 tu = __fadd2_rd(ul, bias), tv = __fadd2_rd(vl, bias);
    const float2 fx = sub2(ul, __fadd2_rn(tu, nbias)), fy = sub2(vl, __fadd2_rn(tv, nbias));
    float2 t00, t01, t10, t11;
    {
        const unsigned x0 = min((unsigned)(ub + __float_as_int(tu.x)), (unsigned)(w - 2));
        const unsigned y0 = min((unsigned)(vb + __float_as_int(tv.x)), (unsigned)(h - 2));
        const unsigned o = y0 * (unsigned)w + x0;   // w h < 2^32: make_coef_group
        MVS_BOUND((long long)o + w + 1 < (long long)h * w);
        t00.x = tap<F16>(img, o);
        t01.x = tap<F16>(img, (long long)o + 1);
        t10.x = tap<F16>(img1, o);
        t11.x = tap<F16>(img1, (long long)o + 1);
    }
    {
        const unsigned x0 = min((unsigned)(ub + __float_as_int(tu.y)), (unsigned)(w - 2));
        const unsigned y0 = min((unsigned)(vb + __float_as_int(tv.y)), (unsigned)(h - 2));
        const unsigned o = y0 * (unsigned)w + x0;
        MVS_BOUND((long long)o + w + 1 < (long long)h * w);
        t00.y = tap<F16>(img, o);
        t01.y = tap<F16>(img, (long long)o + 1);
        t10.y = tap<F16>(img1, o);
        t11.y = tap<F16>(img1, (long long)o + 1);
    }
    const float2 top = __ffma2_rn(fx, sub2(t01, t00), t00);
    const float2 bot = __ffma2_rn(fx, sub2(t11, t10), t10);
    return __ffma2_rn(fy, sub2(bot, top), top);
}

// ---- ray path: per-pixel inverse depth and world ray, FP64 projection with radial distortion and
// FP64 bilinear (_sweep.h:49-80). The reference's point is X = b + (1 / inv) R ray; only its ratios
// enter, so it is formed times inv, X = inv b + R ray, with no reciprocal of the depth, and x / z and
// y / z share one reciprocal of z. What bounds it on an SM is the FP64 pipe (64 lanes a clock, ~40
// operations a sample) and the conversion unit (16 lanes a clock: 3 ray components, 4 taps, the
// inverse depth and the result), so the integer tap position comes from an addition rounded toward
// -inf instead of two conversions, and the bounds are compared as integers. (The order of the float64
// operations is therefore not the reference's: samples differ from it in their last bits and depth
// maps by up to 1.3e-5 relative (1600 x 1200 and 4000 x 3000 views), with the same error against exact
// arithmetic.)

// The source position of one sample: offset of the top-left tap (0 when invalid) and the fractions.
struct RayTap {
    double fx, fy;
    long long o;
    bool ok;
};

template <bool PINHOLE>
__device__ __forceinline__ RayTap ray_tap(const SrcGeo& g, float inv, float rx, float ry, float rz) {
    // inv = +-inf is depth 0: the point is b, whatever the (finite) ray
    const bool at_centre = fabsf(inv) == INFINITY;
    const float m = at_centre ? 0.f : 1.f, af = at_centre ? 1.f : inv;
    const double a = (double)af, dx = (double)__fmul_rn(rx, m), dy = (double)__fmul_rn(ry, m),
                 dz = (double)__fmul_rn(rz, m);
    const double X = __fma_rn(a, g.b[0], __fma_rn(g.m[2], dz, __fma_rn(g.m[1], dy, __dmul_rn(g.m[0], dx))));
    const double Y = __fma_rn(a, g.b[1], __fma_rn(g.m[5], dz, __fma_rn(g.m[4], dy, __dmul_rn(g.m[3], dx))));
    const double Z = __fma_rn(a, g.b[2], __fma_rn(g.m[8], dz, __fma_rn(g.m[7], dy, __dmul_rn(g.m[6], dx))));
    const double iz = rcp_newton(Z);
    const double nx = __dmul_rn(X, iz), ny = __dmul_rn(Y, iz);
    double dd = g.f;   // a pinhole's factor f (1 + r2 (0 + r2 (0 + r2 0))) is exactly f
    if (!PINHOLE) {
        const double r2 = __fma_rn(nx, nx, __dmul_rn(ny, ny));
        dd = __dmul_rn(g.f, __fma_rn(r2, __fma_rn(r2, __fma_rn(r2, g.k3, g.k2), g.k1), 1.0));
    }
    const double u = __fma_rn(dd, nx, g.cx), v = __fma_rn(dd, ny, g.cy);
    // camera depth Z / inv > 1e-6: Z - 1e-6 inv has the sign of inv
    const double t = __fma_rn(-1e-6, a, Z);
    RayTap s;
    s.ok = (__double2hiint(t) ^ __double2hiint(a)) >= 0 && af != 0.f;
    // 0 <= u <= w - 1.001 on the bit patterns as unsigned integers: a negative or NaN u is above
    // every limit (NaN hypotheses count as invalid; the reference leaves them undefined)
    s.ok = s.ok && (unsigned long long)__double_as_longlong(u) <= (unsigned long long)__double_as_longlong((double)g.w - 1.001) &&
           (unsigned long long)__double_as_longlong(v) <= (unsigned long long)__double_as_longlong((double)g.h - 1.001);
    // floor: u + 1.5 * 2^52 rounded toward -inf holds floor(u) in its low word
    const double tu = __dadd_rd(u, 6755399441055744.0), tv = __dadd_rd(v, 6755399441055744.0);
    s.fx = __dsub_rn(u, __dsub_rn(tu, 6755399441055744.0));
    s.fy = __dsub_rn(v, __dsub_rn(tv, 6755399441055744.0));
    s.o = s.ok ? (long long)__double2loint(tv) * g.w + __double2loint(tu) : 0;
    MVS_BOUND(s.o >= 0 && s.o + g.w + 1 < (long long)g.h * g.w);
    return s;
}

__device__ __forceinline__ float ray_value(const RayTap& s, float t00, float t01, float t10, float t11) {
    const double gx = __dsub_rn(1.0, s.fx), gy = __dsub_rn(1.0, s.fy);
    const double top = __fma_rn((double)t01, s.fx, __dmul_rn((double)t00, gx));
    const double bot = __fma_rn((double)t11, s.fx, __dmul_rn((double)t10, gx));
    const float val = (float)__fma_rn(bot, s.fy, __dmul_rn(top, gy));
    return s.ok && isfinite(val) ? val : qnan();
}

// Stage A of the ray path: a thread keeps halo column c and rows seg, seg + SEG, ... as in the plane
// path, and its share of the 2R right-hand columns; `inv` holds its samples' inverse depths for
// this hypothesis (NaN: no sample), in registers because every source uses them (reloading base
// and step per source: 4000 x 3000, R = 3, 22.7 against 15.1 ms). GROUP samples are in flight
// together. Against one sample at a time with four conversions more and two divisions:
// depth_map's three sweeps take 29.5 -> 15.1 ms at 4000 x 3000 (8 sources, R = 3), 5.0 -> 2.5 ms at
// 1600 x 1200 (4 sources, R = 5), 0.99 -> 0.19 ms at 320 x 240 (most of it more, smaller chunks).
template <int R, int TH>
struct RayShare {
    static constexpr int NT = TileShape<TH>::NT, SEG = TileShape<TH>::SEG, HR = Geom<R, TH>::HR;
    static constexpr int MR = (HR + SEG - 1) / SEG;                        // samples in the own column
    static constexpr int XW = R > 0 ? 2 * R : 1, XS = 2 * R * HR, PX = (XS + NT - 1) / NT;
    static constexpr int NS = MR + PX;
    // halo position of sample k; false: a surplus sample (past the tile)
    static __device__ __forceinline__ bool at(int k, int tid, int& hy, int& hc) {
        if (k < MR) {
            hy = tid / TW + k * SEG;
            hc = tid % TW;
            return (k + 1) * SEG <= HR || hy < HR;
        }
        const int e = tid + (k - MR) * NT;
        hy = e / XW;
        hc = TW + (e - hy * XW);
        return (k - MR + 1) * NT <= XS || e < XS;
    }
};

template <int R, int TH, bool PINHOLE>
__device__ __forceinline__ void stage_a_ray(const SweepParams& p, const SrcGeo& g, const float (&inv)[RayShare<R, TH>::NS],
                                            int tx, int ty, int tid, float* sJ, bool& any_invalid, bool& any_valid) {
    using S = RayShare<R, TH>;
    using G = Geom<R, TH>;
    constexpr int GROUP = 4;
    const long long HW = (long long)p.H * p.W;
    const float* img = reinterpret_cast<const float*>(g.img);
    const float* img1 = img + g.w;
#pragma unroll
    for (int k0 = 0; k0 < S::NS; k0 += GROUP) {
        RayTap tap[GROUP];
        float t00[GROUP], t01[GROUP], t10[GROUP], t11[GROUP];
#pragma unroll
        for (int q = 0; q < GROUP; ++q) {
            if (k0 + q >= S::NS) continue;
            int hy, hc;
            S::at(k0 + q, tid, hy, hc);
            // out-of-image and surplus samples (inv = NaN) read a ray of the image
            const int gy = min(max(ty - R + hy, 0), p.H - 1), gx = min(max(tx - R + hc, 0), p.W - 1);
            const float* r = p.ray + ((long long)gy * p.W + gx);
            tap[q] = ray_tap<PINHOLE>(g, inv[k0 + q], __ldg(r), __ldg(r + HW), __ldg(r + 2 * HW));
        }
#pragma unroll
        for (int q = 0; q < GROUP; ++q) {
            if (k0 + q >= S::NS) continue;
            const float *a = img + tap[q].o, *b = img1 + tap[q].o;
            t00[q] = __ldg(a);
            t01[q] = __ldg(a + 1);
            t10[q] = __ldg(b);
            t11[q] = __ldg(b + 1);
        }
#pragma unroll
        for (int q = 0; q < GROUP; ++q) {
            if (k0 + q >= S::NS) continue;
            const float J = ray_value(tap[q], t00[q], t01[q], t10[q], t11[q]);
            int hy, hc;
            if (S::at(k0 + q, tid, hy, hc)) {
                MVS_BOUND(hy * G::JP + (G::RA - R) + hc < G::HR * G::JP);
                any_invalid |= J != J;
                any_valid |= J == J;
                sJ[hy * G::JP + (G::RA - R) + hc] = J;
            }
        }
    }
}

// The plane map of one (hypothesis, source, tile), composed in FP64 and rounded once (Coef),
// by the 4 lanes of an aligned lane group: lane k tests corner k of the halo rectangle, lane 0
// also forms the map, so the four corner tests' divisions run in parallel. A projective map whose
// depth stays positive maps the halo rectangle onto the convex hull of its corner images, so four
// corners strictly inside (a 1e-3 px margin absorbs the FP32 evaluation error of ~1e-5 px) put
// every sample inside, and four corners beyond the same image border put every sample outside:
// that source's NCC is -1 at every pixel of the tile and none of its stages run. Every lane of the
// calling warps must call it (width-4 shuffles); `write` selects the groups that store their
// source's Coef.
__device__ inline void make_coef_group(Coef& c, const SrcGeo& g, float inv, int ox, int oy, int a_lo, int a_hi, int b_lo,
                                       int b_hi, bool write) {
    const int k = threadIdx.x & 3;
    const double d = 1.0 / (double)inv;
    double g0[3], g1[3], g2[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        g1[q] = d * g.m[3 * q + 0];
        g2[q] = d * g.m[3 * q + 1];
        g0[q] = d * (g.m[3 * q + 0] * (double)ox + g.m[3 * q + 1] * (double)oy + g.m[3 * q + 2]) + g.b[q];
    }
    const double Z0 = g0[2];
    const bool norm = fabs(Z0) > 1e-9;
    // corner k of the halo rectangle's part inside the reference image (the rest has no samples)
    const double ca = (double)((k & 1) ? a_hi : a_lo), cb = (double)((k & 2) ? b_hi : b_lo);
    const double Xc = g0[0] + ca * g1[0] + cb * g2[0];
    const double Yc = g0[1] + ca * g1[1] + cb * g2[1];
    const double Zc = g0[2] + ca * g1[2] + cb * g2[2];
    const double uc = g.f * Xc / Zc + g.cx, vc = g.f * Yc / Zc + g.cy;
    int in = Zc > 1e-5 && uc >= 1e-3 && vc >= 1e-3 && uc <= (double)g.w - 1.001 - 1e-3 &&
             vc <= (double)g.h - 1.001 - 1e-3;
    // bits 0-3: this corner is in front and beyond the left / right / top / bottom border
    int out = 0;
    if (Zc > 1e-5) {
        out = (uc <= -1e-3 ? 1 : 0) | (uc >= (double)g.w - 1.001 + 1e-3 ? 2 : 0) | (vc <= -1e-3 ? 4 : 0) |
              (vc >= (double)g.h - 1.001 + 1e-3 ? 8 : 0);
    }
    in &= __shfl_xor_sync(0xffffffffu, in, 1, 4);
    in &= __shfl_xor_sync(0xffffffffu, in, 2, 4);
    out &= __shfl_xor_sync(0xffffffffu, out, 1, 4);
    out &= __shfl_xor_sync(0xffffffffu, out, 2, 4);
    if (k != 0 || !write) return;
    const double zs = norm ? Z0 : 1.0;
    const double rzs = 1.0 / zs;
    double U0 = 0.0, V0 = 0.0;
    if (norm) {
        const double u00 = g.f * g0[0] * rzs + g.cx, v00 = g.f * g0[1] * rzs + g.cy;
        if (isfinite(u00)) U0 = fmin(fmax(floor(u00), -1048576.0), 1048576.0);
        if (isfinite(v00)) V0 = fmin(fmax(floor(v00), -1048576.0), 1048576.0);
    }
    const double au = g.cx - U0, av = g.cy - V0;
    c.nu0 = dup2((float)((g.f * g0[0] + au * g0[2]) * rzs));
    c.nu1 = dup2((float)((g.f * g1[0] + au * g1[2]) * rzs));
    c.nu2 = dup2((float)((g.f * g2[0] + au * g2[2]) * rzs));
    c.nv0 = dup2((float)((g.f * g0[1] + av * g0[2]) * rzs));
    c.nv1 = dup2((float)((g.f * g1[1] + av * g1[2]) * rzs));
    c.nv2 = dup2((float)((g.f * g2[1] + av * g2[2]) * rzs));
    c.dz0 = dup2((float)(g0[2] * rzs));
    c.dz1 = dup2((float)(g1[2] * rzs));
    c.dz2 = dup2((float)(g2[2] * rzs));
    c.zs = (float)zs;
    c.lo_u = (float)(-U0);
    c.lo_v = (float)(-V0);
    c.hi_u = (float)(((double)g.w - 1.001) - U0);
    c.hi_v = (float)(((double)g.h - 1.001) - V0);
    c.U0 = (int)U0;
    c.V0 = (int)V0;
    // (the inside path's tap offsets are 32-bit)
    const bool narrow = (long long)g.w * g.h < (1LL << 32);
    c.inside = !norm ? MAP_MIXED : (in && narrow ? MAP_INSIDE : (out ? MAP_OUTSIDE : MAP_MIXED));
}

// Stage B: horizontal window sums of (V, J, J^2, J I) for one 16-column row segment per thread:
// products formed once per input, running sums along the segment, one float4 per output.
// WITHV = false when every sample is valid: the count column is not formed (it would be k).
template <int R, bool WITHV, int TH = TH_DEFAULT>
__device__ __forceinline__ void stage_b(const float* sJ, const float* sI, float4* sH, int tid) {
    using G = Geom<R, TH>;
    constexpr int RA = G::RA, HR = G::HR, JP = G::JP, P = G::P, NSEG = G::NSEG, NIN = G::NIN;
    if (tid >= HR * NSEG) return;
    // consecutive threads take consecutive rows of one segment: a quarter-warp's 16-byte loads then
    // start (19 hy + 4 sg) mod 8 float4 units into the bank space - 8 distinct groups (JP = 76)
    const int sg = tid / HR, hy = tid - sg * HR;
    MVS_BOUND(hy < HR && P * sg + P <= TW && hy * JP + P * sg + NIN <= HR * JP);
    const float4* jr = reinterpret_cast<const float4*>(sJ + hy * JP + P * sg);
    const float4* ir = reinterpret_cast<const float4*>(sI + hy * JP + P * sg);
    float v[NIN], s1[NIN], s2[NIN], s3[NIN];
#pragma unroll
    for (int q = 0; q < NIN / 4; ++q) {
        float4 a = jr[q];
        const float4 b = ir[q];
        if constexpr (WITHV) {
            float* jv = &a.x;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool ok = finite_value(jv[u]);
                jv[u] = ok ? jv[u] : 0.f;
                v[4 * q + u] = ok ? 1.f : 0.f;
            }
        }
        const float2 j0 = make_float2(a.x, a.y), j1 = make_float2(a.z, a.w);
        const float2 p0 = __fmul2_rn(j0, j0), p1 = __fmul2_rn(j1, j1);
        const float2 c0 = __fmul2_rn(j0, make_float2(b.x, b.y)), c1 = __fmul2_rn(j1, make_float2(b.z, b.w));
        s1[4 * q] = a.x; s1[4 * q + 1] = a.y; s1[4 * q + 2] = a.z; s1[4 * q + 3] = a.w;
        s2[4 * q] = p0.x; s2[4 * q + 1] = p0.y; s2[4 * q + 2] = p1.x; s2[4 * q + 3] = p1.y;
        s3[4 * q] = c0.x; s3[4 * q + 1] = c0.y; s3[4 * q + 2] = c1.x; s3[4 * q + 3] = c1.y;
    }
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int t = RA - R; t <= RA + R; ++t) {
        if constexpr (WITHV) a0 = __fadd_rn(a0, v[t]);
        a1 = __fadd_rn(a1, s1[t]);
        a2 = __fadd_rn(a2, s2[t]);
        a3 = __fadd_rn(a3, s3[t]);
    }
    // hs_index(hy, P sg + j) = hy TW + P sg + (j ^ kx): the segment's columns share (col >> 4) = sg
    float4* row = sH + hy * TW + P * sg;
    const int kx = (sg + hy) & 7;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        if (j > 0) {
            const int tn = RA + R + j, to = RA - R + j - 1;
            if constexpr (WITHV) a0 = __fadd_rn(a0, __fsub_rn(v[tn], v[to]));
            a1 = __fadd_rn(a1, __fsub_rn(s1[tn], s1[to]));
            a2 = __fadd_rn(a2, __fsub_rn(s2[tn], s2[to]));
            a3 = __fadd_rn(a3, __fsub_rn(s3[tn], s3[to]));
        }
        row[j ^ kx] = make_float4(a0, a1, a2, a3);
    }
}

// Inserts one source's NCC into a pixel's sorted list (top list: descending; bottom list: ascending).
template <int KMAX>
__device__ __forceinline__ void topk_insert(float (&list)[KMAX], float& total, float ncc, bool bottom, int nlist) {
    if (bottom) total = __fadd_rn(total, ncc);
    float x = ncc;
#pragma unroll
    for (int q = 0; q < KMAX; ++q) {
        if (q < nlist) {
            const float hi = fmaxf(list[q], x), lo = fminf(list[q], x);
            list[q] = bottom ? lo : hi;
            x = bottom ? hi : lo;
        }
    }
}

// Stage C for one thread: vertical running sums down column c (rows y0 .. y0 + ROWS - 1), ZNCC,
// insertion into the per-pixel top-k lists. WITHV = false: every window count is k^2.
template <int R, int KMAX, bool WITHV, int TH = TH_DEFAULT>
__device__ __forceinline__ void stage_c(const float4* sH, int c, int y0, const float* mu, const float* rsd,
                                        float (&topk)[ROWS][KMAX], float* total, bool bottom, int nlist) {
    constexpr int K = 2 * R + 1;
    const float k2 = (float)(K * K), inv_k2 = 1.0f / (float)(K * K);
    // y0 is a multiple of 8 (ROWS = 8), so hs_index(y0 + t, c) = (y0 + t) TW + sw[t & 7]
    static_assert(ROWS % 8 == 0, "stage C rows must start on a multiple of 8");
    int sw[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) sw[k] = c ^ (((c >> 4) + k) & 7);
    const float4* col = sH + y0 * TW;
    MVS_BOUND(y0 + ROWS + 2 * R <= (Geom<R, TH>::HR) && c < TW);
    // (count, J) and (J^2, J I) as packed pairs: the halves of a 16-byte load
    float2 s01 = dup2(0.f), s23 = dup2(0.f);
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const float4 h = col[t * TW + sw[t & 7]];
        s01 = __fadd2_rn(s01, make_float2(h.x, h.y));
        s23 = __fadd2_rn(s23, make_float2(h.z, h.w));
    }
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        if (j > 0) {
            const float4 hn = col[(j + 2 * R) * TW + sw[(j + 2 * R) & 7]];
            const float4 ho = col[(j - 1) * TW + sw[(j - 1) & 7]];
            s01 = __fadd2_rn(s01, sub2(make_float2(hn.x, hn.y), make_float2(ho.x, ho.y)));
            s23 = __fadd2_rn(s23, sub2(make_float2(hn.z, hn.w), make_float2(ho.z, ho.w)));
        }
        const float cv = s01.x, cj = s01.y;
        float ncc;
        if (WITHV && cv * 10.f <= 9.f * k2) {
            ncc = -1.f;
        } else {
            const float rc = (!WITHV || cv == k2) ? inv_k2 : __frcp_rn(cv);
            const float2 m = __fmul2_rn(s23, dup2(rc));
            const float mj = __fmul_rn(cj, rc), m2 = m.x, mij = m.y;
            const float var = __fsub_rn(m2, __fmul_rn(mj, mj));
            const float rsdj = var > 1e-6f ? rsqrt_ftz(var) : 1000.f;
            ncc = __fmul_rn(__fsub_rn(mij, __fmul_rn(mu[j], mj)), __fmul_rn(rsd[j], rsdj));
            ncc = clip_ncc(ncc);
        }
        topk_insert<KMAX>(topk[j], total[j], ncc, bottom, nlist);
    }
}

// ---- float64 window sums (MVS_PREC_FP64_SUMS): the reference's arithmetic for the sums
// (_sweep.h:85-178): the products J J and J I formed in float32 (float times float, as there),
// horizontal window sums accumulated in float64 - the new column added, then the old one
// subtracted - and stored rounded to float32, as the reference stores its hs rows; vertical sums
// in float64 (add, then subtract), the moments scaled by 1 / k^2 and divided by the scaled count,
// the count gate, variance and NCC in float64 (om_sw_ncc_row), the NCC rounded to float32 once.
// On bright low-texture windows, where the NCC divides by sd_ref * sd_src ~ 1e-3, float32 running
// sums differ from the reference by up to ~1e-3; these track it to the last float32 bit or so.

template <int R, bool WITHV, int TH = TH_DEFAULT>
__device__ __forceinline__ void stage_b64(const float* sJ, const float* sI, float4* sH, int tid) {
    using G = Geom<R, TH>;
    constexpr int RA = G::RA, HR = G::HR, JP = G::JP, P = G::P, NSEG = G::NSEG, NIN = G::NIN;
    if (tid >= HR * NSEG) return;
    const int sg = tid / HR, hy = tid - sg * HR;
    MVS_BOUND(hy < HR && P * sg + P <= TW && hy * JP + P * sg + NIN <= HR * JP);
    const float4* jr = reinterpret_cast<const float4*>(sJ + hy * JP + P * sg);
    const float4* ir = reinterpret_cast<const float4*>(sI + hy * JP + P * sg);
    float v[NIN], jz[NIN], q2[NIN], q3[NIN];
#pragma unroll
    for (int q = 0; q < NIN / 4; ++q) {
        const float4 a = jr[q], b = ir[q];
        const float jv[4] = {a.x, a.y, a.z, a.w}, iv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int t = 4 * q + u;
            float x = jv[u];
            if constexpr (WITHV) {
                const bool ok = finite_value(x);
                x = ok ? x : 0.f;
                v[t] = ok ? 1.f : 0.f;
            }
            jz[t] = x;
            q2[t] = __fmul_rn(x, x);
            q3[t] = __fmul_rn(x, iv[u]);
        }
    }
    float a0 = 0.f;                       // counts are small integers: exact in float32
    double a1 = 0.0, a2 = 0.0, a3 = 0.0;
#pragma unroll
    for (int t = RA - R; t <= RA + R; ++t) {
        if constexpr (WITHV) a0 = __fadd_rn(a0, v[t]);
        a1 = __dadd_rn(a1, (double)jz[t]);
        a2 = __dadd_rn(a2, (double)q2[t]);
        a3 = __dadd_rn(a3, (double)q3[t]);
    }
    float4* row = sH + hy * TW + P * sg;
    const int kx = (sg + hy) & 7;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        if (j > 0) {
            const int tn = RA + R + j, to = RA - R + j - 1;
            if constexpr (WITHV) a0 = __fadd_rn(a0, __fsub_rn(v[tn], v[to]));
            a1 = __dsub_rn(__dadd_rn(a1, (double)jz[tn]), (double)jz[to]);
            a2 = __dsub_rn(__dadd_rn(a2, (double)q2[tn]), (double)q2[to]);
            a3 = __dsub_rn(__dadd_rn(a3, (double)q3[tn]), (double)q3[to]);
        }
        row[j ^ kx] = make_float4(a0, (float)a1, (float)a2, (float)a3);
    }
}

// `sdv` holds the reference's window deviation itself (not its reciprocal) in this mode.
template <int R, int KMAX, bool WITHV, int TH = TH_DEFAULT>
__device__ __forceinline__ void stage_c64(const float4* sH, int c, int y0, const float* mu, const float* sdv,
                                          float (&topk)[ROWS][KMAX], float* total, bool bottom, int nlist) {
    constexpr int K = 2 * R + 1;
    const double kkd = 1.0 / (double)(K * K);
    static_assert(ROWS % 8 == 0, "stage C rows must start on a multiple of 8");
    int sw[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) sw[k] = c ^ (((c >> 4) + k) & 7);
    const float4* col = sH + y0 * TW;
    MVS_BOUND(y0 + ROWS + 2 * R <= (Geom<R, TH>::HR) && c < TW);
    float cv = 0.f;
    double cj = 0.0, cjj = 0.0, cji = 0.0;
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const float4 h = col[t * TW + sw[t & 7]];
        if constexpr (WITHV) cv = __fadd_rn(cv, h.x);
        cj = __dadd_rn(cj, (double)h.y);
        cjj = __dadd_rn(cjj, (double)h.z);
        cji = __dadd_rn(cji, (double)h.w);
    }
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        if (j > 0) {
            const float4 hn = col[(j + 2 * R) * TW + sw[(j + 2 * R) & 7]];
            const float4 ho = col[(j - 1) * TW + sw[(j - 1) & 7]];
            if constexpr (WITHV) cv = __fadd_rn(cv, __fsub_rn(hn.x, ho.x));
            cj = __dsub_rn(__dadd_rn(cj, (double)hn.y), (double)ho.y);
            cjj = __dsub_rn(__dadd_rn(cjj, (double)hn.z), (double)ho.z);
            cji = __dsub_rn(__dadd_rn(cji, (double)hn.w), (double)ho.w);
        }
        float ncc;
        const double cov = __dmul_rn(WITHV ? (double)cv : (double)(K * K), kkd);
        if (cov <= 0.9) {
            ncc = -1.f;
        } else {
            const double mj = __ddiv_rn(__dmul_rn(cj, kkd), cov), m2 = __ddiv_rn(__dmul_rn(cjj, kkd), cov);
            const double mij = __ddiv_rn(__dmul_rn(cji, kkd), cov);
            const double var = __dsub_rn(m2, __dmul_rn(mj, mj));
            const double sdj = var > 1e-6 ? __dsqrt_rn(var) : 1e-3;
            double x = __ddiv_rn(__dsub_rn(mij, __dmul_rn((double)mu[j], mj)), __dmul_rn((double)sdv[j], sdj));
            x = x > 1.0 ? 1.0 : (x < -1.0 ? -1.0 : x);
            ncc = (float)x;
        }
        topk_insert<KMAX>(topk[j], total[j], ncc, bottom, nlist);
    }
}

// ---- compensated window sums (MVS_PREC_FP32_COMP / MVS_PREC_FP16_COMP)
//
// A bright, low-texture window (grey ~1.5, deviations ~0.05) makes the plain form's moments
// m2 - mj^2 and mij - mu mj differences of numbers ~2.25 that agree to ~3 digits, so float32
// rounding of the sums (and of the reference statistics) reaches the NCC a thousand-fold. This form
// removes the large common part before anything is summed: the tile's reference values and every
// warped source value are shifted by one pivot per tile (the mean reference value of the tile's
// pixels), the window sums of the shifted values are accumulated with Kahan compensation in the
// vertical direction (the variance and covariance terms), and the reference window statistics are
// formed from the shifted tile (zero padding outside the image, divided by k^2, floor 1e-6 on the
// variance: the reference's definitions). With I' = I - p and J' = J - p:
//   var(J) = E[J'^2] - E[J']^2,   E[IJ] - mu E[J] = E[I'J'] - mu' E[J'] + p (E[I'] - mu'),
// mu' = mu - p; E[] over the window's valid samples. When every sample of the tile is valid the
// windows are full and E[I'] = mu' exactly, so the last term is zero and is not formed; otherwise
// the masked sum of I' is accumulated as a fifth quantity (the counts then move to a byte array).

template <int R, bool WITHV, int TH = TH_DEFAULT>
__device__ __forceinline__ void stage_b_cmp(const float* sJ, const float* sI, float4* sH, unsigned char* sV, int tid) {
    using G = Geom<R, TH>;
    constexpr int RA = G::RA, HR = G::HR, JP = G::JP, P = G::P, NSEG = G::NSEG, NIN = G::NIN;
    if (tid >= HR * NSEG) return;
    const int sg = tid / HR, hy = tid - sg * HR;
    MVS_BOUND(hy < HR && P * sg + P <= TW && hy * JP + P * sg + NIN <= HR * JP);
    const float4* jr = reinterpret_cast<const float4*>(sJ + hy * JP + P * sg);
    const float4* ir = reinterpret_cast<const float4*>(sI + hy * JP + P * sg);
    float v[NIN], s0[NIN], s1[NIN], s2[NIN], s3[NIN];
#pragma unroll
    for (int q = 0; q < NIN / 4; ++q) {
        const float4 a = jr[q], b = ir[q];
        const float jv[4] = {a.x, a.y, a.z, a.w}, iv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int t = 4 * q + u;
            float jz = jv[u];
            if constexpr (WITHV) {
                const bool ok = finite_value(jz);
                jz = ok ? jz : 0.f;
                v[t] = ok ? 1.f : 0.f;
                s0[t] = ok ? iv[u] : 0.f;
            }
            s1[t] = jz;
            s2[t] = __fmul_rn(jz, jz);
            s3[t] = __fmul_rn(jz, iv[u]);
        }
    }
    float a0 = 0.f, a4 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int t = RA - R; t <= RA + R; ++t) {
        if constexpr (WITHV) {
            a0 = __fadd_rn(a0, v[t]);
            a4 = __fadd_rn(a4, s0[t]);
        }
        a1 = __fadd_rn(a1, s1[t]);
        a2 = __fadd_rn(a2, s2[t]);
        a3 = __fadd_rn(a3, s3[t]);
    }
    float4* row = sH + hy * TW + P * sg;
    unsigned char* crow = sV + hy * TW + P * sg;
    const int kx = (sg + hy) & 7;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        if (j > 0) {
            const int tn = RA + R + j, to = RA - R + j - 1;
            if constexpr (WITHV) {
                a0 = __fadd_rn(a0, __fsub_rn(v[tn], v[to]));
                a4 = __fadd_rn(a4, __fsub_rn(s0[tn], s0[to]));
            }
            a1 = __fadd_rn(a1, __fsub_rn(s1[tn], s1[to]));
            a2 = __fadd_rn(a2, __fsub_rn(s2[tn], s2[to]));
            a3 = __fadd_rn(a3, __fsub_rn(s3[tn], s3[to]));
        }
        row[j ^ kx] = make_float4(a4, a1, a2, a3);
        if constexpr (WITHV) crow[j] = (unsigned char)a0;
    }
}

// Kahan step: s += x with the running compensation c (s - c is the better estimate).
__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
}

// `mu` holds the pivoted window mean mu' = mu - p and `rsd` the reciprocal window deviation, both
// formed from the pivoted reference tile.
template <int R, int KMAX, bool WITHV, int TH = TH_DEFAULT>
__device__ __forceinline__ void stage_c_cmp(const float4* sH, const unsigned char* sV, int c, int y0, const float* mu,
                                            const float* rsd, float pv, float (&topk)[ROWS][KMAX], float* total,
                                            bool bottom, int nlist) {
    constexpr int K = 2 * R + 1;
    const float k2 = (float)(K * K), inv_k2 = 1.0f / (float)(K * K);
    static_assert(ROWS % 8 == 0, "stage C rows must start on a multiple of 8");
    int sw[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) sw[k] = c ^ (((c >> 4) + k) & 7);
    const float4* col = sH + y0 * TW;
    MVS_BOUND(y0 + ROWS + 2 * R <= (Geom<R, TH>::HR) && c < TW);
    const unsigned char* ccol = sV + y0 * TW + c;
    float cv = 0.f, ci = 0.f, cj = 0.f, cjj = 0.f, cji = 0.f;
    float ej = 0.f, ejj = 0.f, eji = 0.f;            // Kahan compensations
#pragma unroll
    for (int t = 0; t < K; ++t) {
        const float4 h = col[t * TW + sw[t & 7]];
        if constexpr (WITHV) {
            cv = __fadd_rn(cv, (float)ccol[t * TW]);
            ci = __fadd_rn(ci, h.x);
        }
        kahan_add(cj, ej, h.y);
        kahan_add(cjj, ejj, h.z);
        kahan_add(cji, eji, h.w);
    }
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        if (j > 0) {
            const float4 hn = col[(j + 2 * R) * TW + sw[(j + 2 * R) & 7]];
            const float4 ho = col[(j - 1) * TW + sw[(j - 1) & 7]];
            if constexpr (WITHV) {
                cv = __fadd_rn(cv, __fsub_rn((float)ccol[(j + 2 * R) * TW], (float)ccol[(j - 1) * TW]));
                ci = __fadd_rn(ci, __fsub_rn(hn.x, ho.x));
            }
            kahan_add(cj, ej, hn.y);
            kahan_add(cj, ej, -ho.y);
            kahan_add(cjj, ejj, hn.z);
            kahan_add(cjj, ejj, -ho.z);
            kahan_add(cji, eji, hn.w);
            kahan_add(cji, eji, -ho.w);
        }
        float ncc;
        if (WITHV && cv * 10.f <= 9.f * k2) {
            ncc = -1.f;
        } else {
            const float rc = (!WITHV || cv == k2) ? inv_k2 : __frcp_rn(cv);
            const float mj = __fmul_rn(__fsub_rn(cj, ej), rc), m2 = __fmul_rn(__fsub_rn(cjj, ejj), rc);
            const float mij = __fmul_rn(__fsub_rn(cji, eji), rc);
            const float var = __fsub_rn(m2, __fmul_rn(mj, mj));
            const float rsdj = var > 1e-6f ? rsqrt_ftz(var) : 1000.f;
            float cov = __fsub_rn(mij, __fmul_rn(mu[j], mj));
            if (WITHV) cov = __fadd_rn(cov, __fmul_rn(pv, __fsub_rn(__fmul_rn(ci, rc), mu[j])));
            ncc = __fmul_rn(cov, __fmul_rn(rsd[j], rsdj));
            ncc = clip_ncc(ncc);
        }
        topk_insert<KMAX>(topk[j], total[j], ncc, bottom, nlist);
    }
}

// ---- the reference tile by TMA (single-view kernel): one 2D tiled bulk copy per CTA, completed
// on an mbarrier. The copy's box is the tile with its halo, JP x HR floats starting at
// (tx - RA, ty - R): x is a multiple of 4 floats (16 bytes), rows outside the image read as 0,
// as the per-thread loads give.

// Tiles whose reference-tile copy did not complete within the bounded wait (read and cleared by
// mvs_device_faults). The counter exists in the one translation unit that instantiates the TMA
// kernels (sweep.cu defines MVS_SWEEP_TMA_UNIT before including this header); elsewhere a
// REF_TMA instantiation does not compile, so no second, unread copy of the counter can arise.
#ifdef MVS_SWEEP_TMA_UNIT
static __device__ unsigned g_ref_copy_faults;
#endif

constexpr unsigned MVS_WAIT_LIMIT_DEFAULT = 1u << 20;   // try_wait iterations of a bounded wait

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned long long* bar,
                                            unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_addr(dst)), "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// Bounded wait for phase `parity` of an mbarrier: false if it did not complete within `limit`
// try_wait iterations.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity, unsigned limit) {
    for (unsigned it = 0; it < limit; ++it) {
        unsigned done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// One tile x hypothesis range at window radius R. `chunk` >= 0 writes the chunk record `chunk`
// of p.nchunks instead of the caller's state. Explicit _rn arithmetic in stages B and C fixes
// every rounding, so the result never depends on how the compiler scheduled this instance.
// REF_TMA: the reference tile arrives by TMA when p.ref_tma is set (the single-view kernel, whose
// parameters hold the tensor map; `smem` must then be 128-byte aligned).
template <int R, int KMAX, bool PLANES, bool F16, bool REF_TMA = false, bool X64 = false, bool CMP = false,
          int TH = TH_DEFAULT>
__device__ void sweep_tile(const SweepParams& p, int tx, int ty, int pa, int pb, int chunk, float* smem) {
    using G = Geom<R, TH>;
    using WS = WinnerState<R, KMAX, TH>;
    constexpr int NT = TileShape<TH>::NT, SEG = TileShape<TH>::SEG;
    constexpr int K = G::K, RA = G::RA, HR = G::HR, HC = G::HC, JP = G::JP, P = G::P, NSEG = G::NSEG,
                  NIN = G::NIN;
    float* sI = smem;                                  // HR x JP reference (0 outside); TMA destination
    float* sJ = sI + HR * JP;                          // HR x JP warped source (NaN = invalid)
    float4* sH = reinterpret_cast<float4*>(sJ + HR * JP);   // HR x TW (V, J, J^2, J I), swizzled
    const int H = p.H, W = p.W;
    const int tid = threadIdx.x;

    __syncthreads();   // a previous tile of a persistent CTA is done with shared memory
    bool tma = false;
    __shared__ __align__(8) unsigned long long s_ref_bar;
#ifndef MVS_SWEEP_TMA_UNIT
    static_assert(!REF_TMA, "REF_TMA kernels are instantiated in sweep.cu only (it owns the fault counter)");
#else
    if constexpr (REF_TMA) {
        tma = p.ref_tma != 0;
        if (tma && tid == 0) {
            mbar_init(&s_ref_bar, 1);
            tma_load_2d(sI, &p.ref_map, tx - RA, ty - R, &s_ref_bar, (unsigned)(HR * JP * sizeof(float)));
        }
    }
#endif
    for (int e = tid; e < HR * JP; e += NT) {
        if (!tma) {
            const int hy = e / JP, hc = e - hy * JP;
            const int gy = ty - R + hy, gx = tx - RA + hc;
            float v = 0.f;
            if (gy >= 0 && gy < H && gx >= 0 && gx < W) v = __ldg(p.ref + (long long)gy * W + gx);
            sI[e] = v;
        }
        sJ[e] = qnan();
    }

    // winner-take-all state of the tile's pixels: touched once per hypothesis, so it lives in
    // shared memory (planes: best, prev, s_prev_best, s_next_best, idx bits, first score)
    float* sW = reinterpret_cast<float*>(sH + HR * TW);
    Coef* sC = reinterpret_cast<Coef*>(sW + WS::PLANES * TH * TW);
    const int c = tid % TW, seg = tid / TW;
    const float fcol = (float)c, fseg = (float)seg;
    const int gx = tx + c;
    float mu[ROWS], rsd[ROWS];
    const bool to_rec = chunk >= 0;
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        const int ly = seg * ROWS + j, gy = ty + ly;
        const bool in = gx < W && gy < H;
        const long long o = (long long)gy * W + gx;
        // (compensated mode: formed from the pivoted tile below instead)
        mu[j] = in && !CMP ? __ldg(p.mu + o) : 0.f;
        // X64: the deviation itself (stage C divides in float64); else its reciprocal
        rsd[j] = in && !CMP ? (X64 ? __ldg(p.sd + o) : 1.0f / __ldg(p.sd + o)) : 0.f;
        const bool load = in && !to_rec && !p.fresh;
        const int w = ly * TW + c;
        sW[w] = load ? p.best[o] : -2.f;
        sW[TH * TW + w] = load ? p.prev[o] : -2.f;
        sW[2 * TH * TW + w] = load ? p.spb[o] : -2.f;
        sW[3 * TH * TW + w] = load ? p.snb[o] : -2.f;
        sW[4 * TH * TW + w] = __int_as_float(load ? p.idx[o] : -1);
        if constexpr (!WS::FIRST_TO_REC) sW[5 * TH * TW + w] = -2.f;
    }
    const int nsrc = p.n_src, kk = p.kk;
    const bool bottom = KMAX > 2 && p.topk_bottom != 0;   // the 2-entry list is always a top list
    const int nlist = bottom ? nsrc - kk : kk;
    // every halo sample lies inside the reference image (interior tile)
    const bool tile_inside = tx - R >= 0 && ty - R >= 0 && tx + TW + R <= W && ty + TH + R <= H;
#ifdef MVS_SWEEP_TMA_UNIT
    if constexpr (REF_TMA) {
        if (tma) {
            __syncthreads();   // the barrier's initialisation is visible to every thread
            const bool arrived = mbar_wait_bounded(&s_ref_bar, 0, p.wait_limit);
            // a copy that did not complete in time: count it and leave the tile's state untouched.
            // Before the CTA (and its shared memory) goes, wait once more, with the default
            // bound, for the copy that may still be in flight into that memory.
            if (__syncthreads_or(!arrived)) {
                if (tid == 0) {
                    atomicAdd(&g_ref_copy_faults, 1u);
                    mbar_wait_bounded(&s_ref_bar, 0, MVS_WAIT_LIMIT_DEFAULT);
                }
                __syncthreads();
                return;
            }
        }
    }
#endif
    // compensated mode: pivot the reference tile and form its window statistics from it
    float pv = 0.f;
    unsigned char* sV = reinterpret_cast<unsigned char*>(sC + MVS_MAX_SOURCES);   // byte counts
    if constexpr (CMP) {
        __shared__ float red[2 * (NT / 32)];
        __syncthreads();                       // the reference tile is complete (thread loads or TMA)
        float su = 0.f, nn = 0.f;
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const int ly = seg * ROWS + j;
            if (gx < W && ty + ly < H) {
                su = __fadd_rn(su, sI[(ly + R) * JP + RA + c]);
                nn += 1.f;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            su = __fadd_rn(su, __shfl_xor_sync(0xffffffffu, su, o));
            nn += __shfl_xor_sync(0xffffffffu, nn, o);
        }
        if ((tid & 31) == 0) {
            red[tid >> 5] = su;
            red[NT / 32 + (tid >> 5)] = nn;
        }
        __syncthreads();
        su = 0.f;
        nn = 0.f;
        for (int w = 0; w < NT / 32; ++w) {   // every thread sums the warp totals in the same order
            su = __fadd_rn(su, red[w]);
            nn += red[NT / 32 + w];
        }
        pv = nn > 0.f ? __fdiv_rn(su, nn) : 0.f;
        for (int e = tid; e < HR * JP; e += NT) sI[e] = __fsub_rn(sI[e], pv);
        __syncthreads();
        // mu' = sum(I') / k^2 over the zero-padded window (I' = -p outside the image), var =
        // sum(I'^2) / k^2 - mu'^2, sd = sqrt(max(var, 1e-6)): the reference's statistics, pivoted
        const float inv_k2 = 1.0f / (float)(K * K);
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const int ly = seg * ROWS + j;
            float s1 = 0.f, s2 = 0.f;
#pragma unroll 1
            for (int dy = 0; dy < K; ++dy) {
                const float* rowp = sI + (ly + dy) * JP + (RA - R) + c;
#pragma unroll
                for (int dx = 0; dx < K; ++dx) {
                    const float v = rowp[dx];
                    s1 = __fadd_rn(s1, v);
                    s2 = __fmaf_rn(v, v, s2);
                }
            }
            const float m = __fmul_rn(s1, inv_k2);
            const float var = __fsub_rn(__fmul_rn(s2, inv_k2), __fmul_rn(m, m));
            const bool in = gx < W && ty + ly < H;
            mu[j] = in ? m : 0.f;
            rsd[j] = in ? __frcp_rn(__fsqrt_rn(var > 1e-6f ? var : 1e-6f)) : 0.f;
        }
    }

    auto in_image = [&](int hy, int hc) {
        return (unsigned)(ty - R + hy) < (unsigned)H && (unsigned)(tx - R + hc) < (unsigned)W;
    };
    __shared__ unsigned s_reach[2][NT / 32];
    int vote_slot = 0;
    for (int i = pa; i < pb; ++i) {
        float topk[ROWS][KMAX];
        float total[ROWS];
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            total[j] = 0.f;
#pragma unroll
            for (int q = 0; q < KMAX; ++q) topk[j][q] = bottom ? INFINITY : -INFINITY;
        }
        if constexpr (PLANES) {
            __syncthreads();   // the previous hypothesis is done reading sC
            if (tid < 4 * MVS_MAX_SOURCES && (tid >> 5) * 8 < nsrc) {   // the warps that hold a source
                const int sg_ = tid >> 2;
                make_coef_group(sC[sg_ < nsrc ? sg_ : 0], p.src[sg_ < nsrc ? sg_ : 0], p.planes[i - p.i0], tx - R,
                                ty - R, max(R - tx, 0), min(HC, W - (tx - R)) - 1, max(R - ty, 0),
                                min(HR, H - (ty - R)) - 1, sg_ < nsrc);
            }
        }
        // ray path: the inverse depths of the thread's samples, shared by the sources
        float inv[PLANES ? 1 : RayShare<R, TH>::NS];
        if constexpr (!PLANES) {
#pragma unroll
            for (int k = 0; k < RayShare<R, TH>::NS; ++k) {
                int hy, hc;
                const bool own = RayShare<R, TH>::at(k, tid, hy, hc);
                const int hgy = ty - R + hy, hgx = tx - R + hc;
                inv[k] = own && hgy >= 0 && hgy < H && hgx >= 0 && hgx < W ? hyp_value(p, i, hgx, hgy) : qnan();
            }
        }
        // sC ready; first hypothesis: the tile's set-up of sI, sJ and sW too. (Between sources no
        // barrier is needed here: stage B's reads of sJ end before the barrier that follows it, and
        // stage C's reads of sH before the barrier that follows the next stage A.)
        __syncthreads();
        for (int s = 0; s < nsrc; ++s) {
            if constexpr (PLANES) {
                // a source that no sample of the tile reaches: its window counts are 0, its NCC -1
                // (4000 x 3000 view, 8 sources at 80 % / 70 % overlap, 256 planes: 168.9 -> 101.9 ms)
                if (sC[s].inside == MAP_OUTSIDE) {
#pragma unroll
                    for (int j = 0; j < ROWS; ++j) topk_insert<KMAX>(topk[j], total[j], -1.f, bottom, nlist);
                    continue;
                }
            }
            // ---- A: warp the source into the halo tile
            const void* img = p.src[s].img;
            const int sw = p.src[s].w, sh = p.src[s].h;
            bool any_invalid = false, all_valid;
            if constexpr (PLANES) {
                const Coef cf = sC[s];
                if (cf.inside == MAP_INSIDE && tile_inside) {
                    // every sample of the thread gathered before any is stored: the gathers are
                    // independent and in flight together. The thread keeps halo column c and
                    // rows seg, seg + SEG, ... (positions and shared offsets fixed per thread, so
                    // no per-sample index arithmetic); the 2R right-hand halo columns are spread
                    // over all threads. Samples go in pairs; a surplus one (a row or column past
                    // the halo) reads some tap of the image and is not stored.
                    using S = RayShare<R, TH>;
                    constexpr int NP = (S::NS + 1) / 2;
                    const char* img1 = reinterpret_cast<const char*>(img) + (size_t)sw * (F16 ? 2 : 4);
                    const int ub = cf.U0 - 0x4B400000, vb = cf.V0 - 0x4B400000;
                    float2 Jv[NP];
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        float2 a, b;
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            float& aq = q ? a.y : a.x;
                            float& bq = q ? b.y : b.x;
                            if (2 * k + q < S::MR) {
                                aq = fcol;
                                bq = fseg + (float)((2 * k + q) * SEG);
                            } else {
                                int hy, hc;
                                S::at(2 * k + q < S::NS ? 2 * k + q : S::NS - 1, tid, hy, hc);
                                aq = (float)hc;
                                bq = (float)hy;
                            }
                        }
                        Jv[k] = sample_plane_inside2<F16>(cf, img, img1, sw, sh, ub, vb, a, b);
                    }
#pragma unroll
                    for (int k = 0; k < S::NS; ++k) {
                        int hy, hc;
                        if (S::at(k, tid, hy, hc)) {
                            const float J = k & 1 ? Jv[k / 2].y : Jv[k / 2].x;
                            MVS_BOUND(hy * JP + (RA - R) + hc < HR * JP);
                            any_invalid |= !finite_value(J);
                            sJ[hy * JP + (RA - R) + hc] = CMP ? __fsub_rn(J, pv) : J;
                        }
                    }
                } else if (cf.inside == MAP_INSIDE) {
                    // a border tile of the reference whose part of the image maps inside: the same
                    // samples pair by pair (rolled, for its registers: unrolled in the interior form it
                    // cost that form spills, C2 94.5 against 91.4 ms), none outside the image. With
                    // every sample tested as in the form below: 640 x 480, 4 sources, 128 planes 0.92
                    // against 0.87 ms, batch of 8 uneven views 99.7 against 96.2 ms.
                    using S = RayShare<R, TH>;
                    const char* img1 = reinterpret_cast<const char*>(img) + (size_t)sw * (F16 ? 2 : 4);
                    const int ub = cf.U0 - 0x4B400000, vb = cf.V0 - 0x4B400000;
#pragma unroll 1
                    for (int k = 0; k < S::NS; k += 2) {
                        int hy0, hc0, hy1, hc1;
                        const bool own0 = S::at(k, tid, hy0, hc0), own1 = k + 1 < S::NS && S::at(k + 1, tid, hy1, hc1);
                        if (!own1) {
                            hy1 = hy0;
                            hc1 = hc0;
                        }
                        const float2 J = sample_plane_inside2<F16>(cf, img, img1, sw, sh, ub, vb,
                                                                   make_float2((float)hc0, (float)hc1),
                                                                   make_float2((float)hy0, (float)hy1));
                        const float J0 = in_image(hy0, hc0) ? J.x : qnan(), J1 = in_image(hy1, hc1) ? J.y : qnan();
                        if (own0) {
                            MVS_BOUND(hy0 * JP + (RA - R) + hc0 < HR * JP);
                            any_invalid |= !finite_value(J0);
                            sJ[hy0 * JP + (RA - R) + hc0] = CMP ? __fsub_rn(J0, pv) : J0;
                        }
                        if (own1) {
                            MVS_BOUND(hy1 * JP + (RA - R) + hc1 < HR * JP);
                            any_invalid |= !finite_value(J1);
                            sJ[hy1 * JP + (RA - R) + hc1] = CMP ? __fsub_rn(J1, pv) : J1;
                        }
                    }
                } else {
                    constexpr int PER = (HR * HC + NT - 1) / NT;
#pragma unroll 4
                    for (int k = 0; k < PER; ++k) {
                        const int e = tid + k * NT;
                        if (e < HR * HC) {
                            const int hy = e / HC, hc = e - hy * HC;
                            const float J = sample_plane<F16>(cf, img, sw, sh, (float)hc, (float)hy, in_image(hy, hc));
                            MVS_BOUND(hy * JP + (RA - R) + hc < HR * JP);
                            any_invalid |= J != J;
                            sJ[hy * JP + (RA - R) + hc] = CMP ? __fsub_rn(J, pv) : J;
                        }
                    }
                }
            } else {
                static_assert(!CMP, "compensated sums run on the plane path");
                const SrcGeo& g = p.src[s];
                bool any_valid = false;
                if (g.k1 == 0.0 && g.k2 == 0.0 && g.k3 == 0.0)
                    stage_a_ray<R, TH, true>(p, g, inv, tx, ty, tid, sJ, any_invalid, any_valid);
                else
                    stage_a_ray<R, TH, false>(p, g, inv, tx, ty, tid, sJ, any_invalid, any_valid);
                // a source that no sample reached: NCC -1 everywhere, as in the plane path. (The next
                // stage A may write sJ at once: nothing reads it.) The votes alternate between two
                // words, so a thread that runs ahead does not overwrite the one still being read.
                const unsigned vote = (__any_sync(0xffffffffu, any_valid) ? 1u : 0u);
                if ((tid & 31) == 0) s_reach[vote_slot][tid >> 5] = vote;
                all_valid = !__syncthreads_or(any_invalid);
                unsigned reach = 0;
#pragma unroll
                for (int w = 0; w < NT / 32; ++w) reach |= s_reach[vote_slot][w];
                vote_slot ^= 1;
                if (!reach) {
#pragma unroll
                    for (int j = 0; j < ROWS; ++j) topk_insert<KMAX>(topk[j], total[j], -1.f, bottom, nlist);
                    continue;
                }
            }
            // every sample of this (hypothesis, source) valid -> the count is k^2 everywhere and
            // stages B and C skip it (block-wide vote; uniform branch)
            if constexpr (PLANES) all_valid = !__syncthreads_or(any_invalid);
            // ---- B: horizontal window sums of (V, J, J^2, J I), one 16-column row segment per
            // thread: products once per input, running sums along the segment
            if constexpr (CMP) {
                if (all_valid) {
                    stage_b_cmp<R, false, TH>(sJ, sI, sH, sV, tid);
                } else {
                    stage_b_cmp<R, true, TH>(sJ, sI, sH, sV, tid);
                }
            } else if constexpr (X64) {
                if (all_valid) {
                    stage_b64<R, false, TH>(sJ, sI, sH, tid);
                } else {
                    stage_b64<R, true, TH>(sJ, sI, sH, tid);
                }
            } else if (all_valid) {
                stage_b<R, false, TH>(sJ, sI, sH, tid);
            } else {
                stage_b<R, true, TH>(sJ, sI, sH, tid);
            }
            __syncthreads();
            // ---- C: vertical running sums down the column, NCC, top-k insertion
            if constexpr (CMP) {
                if (all_valid) {
                    stage_c_cmp<R, KMAX, false, TH>(sH, sV, c, seg * ROWS, mu, rsd, pv, topk, total, bottom, nlist);
                } else {
                    stage_c_cmp<R, KMAX, true, TH>(sH, sV, c, seg * ROWS, mu, rsd, pv, topk, total, bottom, nlist);
                }
            } else if constexpr (X64) {
                if (all_valid) {
                    stage_c64<R, KMAX, false, TH>(sH, c, seg * ROWS, mu, rsd, topk, total, bottom, nlist);
                } else {
                    stage_c64<R, KMAX, true, TH>(sH, c, seg * ROWS, mu, rsd, topk, total, bottom, nlist);
                }
            } else if (all_valid) {
                stage_c<R, KMAX, false, TH>(sH, c, seg * ROWS, mu, rsd, topk, total, bottom, nlist);
            } else {
                stage_c<R, KMAX, true, TH>(sH, c, seg * ROWS, mu, rsd, topk, total, bottom, nlist);
            }
        }
        // ---- winner-take-all update for hypothesis i
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            float sc = 0.f;
#pragma unroll
            for (int q = 0; q < KMAX; ++q)
                if (q < nlist) sc = __fadd_rn(sc, topk[j][q]);
            if (bottom) sc = __fsub_rn(total[j], sc);
            sc = __fdiv_rn(sc, (float)kk);
            const int w = (seg * ROWS + j) * TW + c;
            MVS_BOUND(w < TH * TW);
            float best = sW[w], prv = sW[TH * TW + w];
            const int id = __float_as_int(sW[4 * TH * TW + w]);
            if (id == i - 1) sW[3 * TH * TW + w] = sc;
            if (sc > best) {
                sW[w] = sc;
                sW[2 * TH * TW + w] = prv;
                sW[3 * TH * TW + w] = -2.f;
                sW[4 * TH * TW + w] = __int_as_float(i);
            }
            sW[TH * TW + w] = sc;
            if constexpr (!WS::FIRST_TO_REC) {
                if (i == pa) sW[5 * TH * TW + w] = sc;
            }
        }
        if constexpr (WS::FIRST_TO_REC) {
            if (to_rec && i == pa) {   // the prev plane holds the chunk's first scores now
#pragma unroll 1
                for (int j = 0; j < ROWS; ++j) {
                    const int gy = ty + seg * ROWS + j;
                    if (gx < W && gy < H)
                        p.rec[(4LL * p.nchunks + chunk) * H * W + (long long)gy * W + gx] =
                            sW[(TH + seg * ROWS + j) * TW + c];
                }
            }
        }
    }

    // ---- write back: caller state (single chunk) or the chunk record
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        const int gy = ty + seg * ROWS + j;
        if (gx >= W || gy >= H) continue;
        const long long o = (long long)gy * W + gx;
        const int w = (seg * ROWS + j) * TW + c;
        if (!to_rec) {
            p.best[o] = sW[w];
            p.prev[o] = sW[TH * TW + w];
            p.spb[o] = sW[2 * TH * TW + w];
            p.snb[o] = sW[3 * TH * TW + w];
            p.idx[o] = __float_as_int(sW[4 * TH * TW + w]);
        } else {
            const long long HW = (long long)H * W;
            const long long plane = (long long)p.nchunks * HW;
            float* rc = p.rec + (long long)chunk * HW + o;
            rc[0] = sW[w];
            rc[plane] = sW[4 * TH * TW + w];
            rc[2 * plane] = sW[2 * TH * TW + w];
            rc[3 * plane] = sW[3 * TH * TW + w];
            if constexpr (!WS::FIRST_TO_REC) rc[4 * plane] = sW[5 * TH * TW + w];
            rc[5 * plane] = sW[TH * TW + w];
        }
    }
}

// Ordered merge of one pixel's chunk records into its state (hypothesis order, first wins).
__device__ __forceinline__ void merge_pixel(long long o, long long HW, int nchunks, int i0, int i1, int ppc,
                                            const float* __restrict__ rec, float& B, float& P, float& SP,
                                            float& SN, int& I) {
    const long long plane = (long long)nchunks * HW;
    for (int ch = 0; ch < nchunks; ++ch) {
        const int a = i0 + ch * ppc, b = min(i1, a + ppc);
        if (a >= b) break;
        const float* r = rec + (long long)ch * HW + o;
        const float cb = r[0];
        const int ci = __float_as_int(r[plane]);
        const float cp = r[2 * plane], cn = r[3 * plane], cf = r[4 * plane], cl = r[5 * plane];
        if (I == a - 1) SN = cf;
        if (cb > B) {
            B = cb;
            I = ci;
            SP = (ci > a) ? cp : P;
            SN = (ci < b - 1) ? cn : -2.f;
        }
        P = cl;
    }
}

// densify.py:354-361: parabola through (idx-1, idx, idx+1) in float32, depth in float64.
__device__ __forceinline__ float finalize_pixel(float inv0, float inv1, int n, float bb, float sp, float sn, int id) {
    const float dinv = n > 1 ? __fsub_rn(inv1, inv0) : 0.f;
    const float den = __fadd_rn(__fsub_rn(sp, __fmul_rn(2.f, bb)), sn);
    const bool interior = id > 0 && id < n - 1 && den < -1e-6f;
    float off = 0.f;
    if (interior) off = __fdiv_rn(__fmul_rn(0.5f, __fsub_rn(sp, sn)), den);
    off = off < -0.5f ? -0.5f : (off > 0.5f ? 0.5f : off);
    const double t = __dadd_rn((double)id, (double)off);
    const double inv = __dadd_rn((double)inv0, __dmul_rn(t, (double)dinv));
    const double m = max_nan(inv, 1e-9);
    return (float)__ddiv_rn(1.0, m);
}

// host-side helpers shared by sweep.cu and batch.cu
inline int tile_height(const mvs_sweep_args* a) { return a->tile_h ? a->tile_h : TH_DEFAULT; }
mvs_status validate_sweep(const mvs_sweep_args* a);
mvs_status fill_params(const mvs_sweep_args* a, SweepParams& p);
int pick_kmax(SweepParams& p);

}  // namespace mvs
