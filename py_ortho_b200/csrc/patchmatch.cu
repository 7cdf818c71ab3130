// Red-black slanted-plane PatchMatch repair (reference: _dense.pm_refine, _dense.pyx:405-666).
//
// This file is compiled with -fmad=false: every float64 expression below is evaluated with one
// rounding per operation in the written order, which is how the reference's C (x86-64, no FMA)
// evaluates it. The float64 mode gives the bits of the reference's pm_refine on every input tested (its
// quotients have an exception, see pm_quot).
//
// Parallel schedule. The reference visits the pixels of one colour ((x + y) % 2) in raster order,
// but every pixel reads only its own plane, pixels of the other colour (all 8 neighbour offsets,
// (+-1, 0), (0, +-1), (+-5, 0), (0, +-5), have odd parity) and static inputs. So all pixels of a
// colour are independent: one thread (or lane group) per pixel per colour pass.
//
// Random trials. The reference draws from ONE xorshift32 stream (_rnd, _dense.pyx:559-563,
// started at seed | 1 per call, :606): 8 draws, in raster order, for every active pixel of the
// colour whose depth is finite once propagation is done (:646-652). Which pixels draw is known
// only after propagation, so a colour pass runs as
//   1. propagation (pm_kernel / pm_lane_kernel, PHASE 0): current plane + 8 neighbour planes;
//      the pixel's best cost, score and a flag "draws" go to per-pass scratch;
//   2. the exclusive prefix count of drawing pixels in raster order (pm_count_kernel,
//      pm_scan_kernel, pm_state_kernel): pixel p's first draw is stream element
//      base + 8 * prefix(p); xorshift32 is linear over GF(2), so its state there is
//      A^(8 prefix(p)) s_base with A the 32 x 32 step matrix, applied as a product of the
//      precomputed powers A^(8 * 2^j) (jump-ahead for F2-linear generators: Haramoto,
//      Matsumoto, Nishimura, Panneton, L'Ecuyer 2008); the pass advances the stream by 8 * total;
//   3. the two random trials (PHASE 1) from the pixel's own stream state.
// The stream state lives on the device from pass to pass (and, with mvs_pm_args.rng_state, from
// call to call), so no step waits for the host.
#include "common.cuh"

#include <algorithm>

namespace mvs {

struct PMStats;

struct PMParams {
    int H, W, S, r, step, top_k, it, colour;
    int last;                           // the window's last offset, -r + m step <= r
    float r2;                           // r r
    int few;                            // at most 400 samples in a window
    double cr0, cr1, cr2, geo_w, geo_tol, dmin, dmax, dd_scale, nn_scale;
    const float* ref;
    const float* ray;
    float* depth;
    float* normal;
    float* score;
    const unsigned char* active;
    unsigned long long* changed;
    double* cost_cache;                // per pixel; NaN = recompute (valid within one call)
    double* score_cache;
    // per colour pass, indexed by the pass's pixel number t = y * ceil(W / 2) + x / 2
    unsigned char* flags;              // bit 0: the pixel draws; bits 1-4: propagation changes
    double* pbest;                     // cost of the plane kept by propagation
    double* psc;                       // its photo score
    const unsigned* pstate;            // xorshift32 state before the pixel's first draw
    unsigned win_smem;                 // dynamic shared bytes of the lane kernel (bounds checks)
    const float* img[MVS_MAX_SOURCES];
    const float* dep[MVS_MAX_SOURCES];
    int iw[MVS_MAX_SOURCES], ih[MVS_MAX_SOURCES];
    int pinhole[MVS_MAX_SOURCES];       // k1 = k2 = k3 = 0
    double par[MVS_MAX_SOURCES * 18];
    double bsrc[MVS_MAX_SOURCES * 3];   // R_s (C_ref - C_s)
    // float64 kernel: the active pixels of this colour (pass pixel numbers in raster order) and their
    // count, both on the device; float32 copies of par and bsrc for the window tests
    const unsigned* list;
    const unsigned* n_list;
    const PMStats* stats;
    float parf[MVS_MAX_SOURCES * 18], bsf[MVS_MAX_SOURCES * 3];
    // float32 lane kernel: per source its 2 x 2 bilinear footprints, quad[y w + x] =
    // (I(y, x), I(y + 1, x), I(y, x + 1), I(y + 1, x + 1)), one 16-byte load per sample whose halves
    // are the operands of the packed interpolation along x
    const float4* quad[MVS_MAX_SOURCES];
};

// ---------------------------------------------------------------- the reference's stream

// _rnd (_dense.pyx:559-563): one xorshift32 step, then the low 24 bits as a uniform in [0, 1).
__host__ __device__ __forceinline__ unsigned xs_step(unsigned s) {
    s ^= s << 13;
    s ^= s >> 17;
    s ^= s << 5;
    return s;
}
__device__ __forceinline__ double xs_draw(unsigned& s) {
    s = xs_step(s);
    return (double)(s & 0xFFFFFFu) / 16777216.0;
}

// A 32 x 32 matrix over GF(2) by columns: col[i] = M e_i, so M s = XOR of col[i] over set bits i.
struct Gf2 {
    unsigned col[32];
};
__host__ __device__ __forceinline__ unsigned gf2_apply(const Gf2& m, unsigned s) {
    unsigned r = 0;
#pragma unroll
    for (int i = 0; i < 32; ++i) r ^= m.col[i] & (0u - ((s >> i) & 1u));
    return r;
}

// Jump table of the stream: t[j] = A^(8 * 2^j), A = one xorshift32 step.
struct PMJump {
    Gf2 t[32];
};

// State after 8 k steps from s.
__device__ __forceinline__ unsigned jump8(const PMJump& J, unsigned s, unsigned k) {
    for (int j = 0; k != 0; ++j, k >>= 1)
        if (k & 1u) s = gf2_apply(J.t[j], s);
    return s;
}

// _proj (_dense.pyx:429-445): world point -> pixel and camera depth.
__device__ __forceinline__ bool pm_proj(const double* p, double X, double Y, double Z, double& u, double& v,
                                        double& z) {
    const double dx = X - p[9], dy = Y - p[10], dz = Z - p[11];
    const double xc = p[0] * dx + p[1] * dy + p[2] * dz;
    const double yc = p[3] * dx + p[4] * dy + p[5] * dz;
    const double zc = p[6] * dx + p[7] * dy + p[8] * dz;
    if (zc <= 1e-6) return false;
    const double nx = xc / zc, ny = yc / zc;
    const double r2 = nx * nx + ny * ny;
    const double dd = p[12] * (1.0 + r2 * (p[13] + r2 * (p[14] + r2 * p[15])));
    u = dd * nx + p[16];
    v = dd * ny + p[17];
    z = zc;
    return true;
}

// _bil (_dense.pyx:448-458); NaN outside [0, w-1.001] x [0, h-1.001] (also for NaN u, v, whose
// behaviour the reference leaves undefined).
__device__ __forceinline__ double pm_bil(const float* im, int w, int h, double u, double v) {
    if (!(u >= 0.0 && v >= 0.0 && u <= (double)w - 1.001 && v <= (double)h - 1.001)) return __longlong_as_double(0x7ff8000000000000LL);
    const int x0 = (int)u, y0 = (int)v;
    const double fx = u - (double)x0, fy = v - (double)y0;
    const long long o = (long long)y0 * w + x0;
    const double a00 = __ldg(im + o), a01 = __ldg(im + o + 1), a10 = __ldg(im + o + w), a11 = __ldg(im + o + w + 1);
    return (a00 * (1.0 - fx) + a01 * fx) * (1.0 - fy) + (a10 * (1.0 - fx) + a11 * fx) * fy;
}

// ---------------------------------------------------------------- float64 evaluation (MVS_PM_FP64)
//
// _pm_cost (_dense.pyx:461-556): every sum, product and comparison that reaches a result is the
// reference's, with its rounding; quotients have pm_quot's exception. What bounds it is the float64 pipe
// (64 lanes a clock per SM), so the work that provably does not reach a result is left out and what is
// shared is formed once:
//   * the geometric term comes first: a candidate whose geometric term alone reaches the pixel's
//     best cost cannot be accepted (the photo term is at least 1 - NCC, see PM_PRUNE), so its windows
//     are not evaluated;
//   * per (candidate, source) the window's four corners are mapped in float32: a source that the
//     whole window misses has NCC -1 (the count gate), one that it hits with a margin needs no
//     per-sample tests, and its reference sums are the pixel's own, formed once per visit;
//   * PM_PASS sources share a sample's world point (one division), and x / z, y / z share one
//     reciprocal; the tap position comes from an addition rounded toward -inf (no conversions);
//   * only active pixels get a thread (PMParams::list).
// Each of a source's sums still accumulates in window order.

// Sources per pass over the window (PM_MIN_BLOCKS has the measurements).
constexpr int PM_PASS = 2;

// What mvs_pm_refine's preparation finds out about its inputs (float bit patterns, all >= 0).
struct PMStats {
    unsigned max_abs;      // largest finite |value| of the reference and the sources
    unsigned ray_bend;     // largest second difference of the ray grid along rows and columns
};

__global__ void __launch_bounds__(256) pm_stats_kernel(const float* __restrict__ im, long long n, PMStats* st) {
    float m = 0.f;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const float v = fabsf(__ldg(im + i));
        if (v <= 3.402823466e38f) m = fmaxf(m, v);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&st->max_abs, __float_as_uint(m));
}

__global__ void __launch_bounds__(256) pm_bend_kernel(const float* __restrict__ ray, int H, int W, PMStats* st) {
    const long long HW = (long long)H * W;
    float m = 0.f;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < HW; i += (long long)gridDim.x * 256) {
        const int y = (int)(i / W), x = (int)(i - (long long)y * W);
        for (int k = 0; k < 3; ++k) {
            const float* r = ray + k * HW + i;
            const float v = __ldg(r);
            if (!(fabsf(v) <= 3.402823466e38f)) m = INFINITY;
            if (x > 0 && x < W - 1) {
                const float d = fabsf((__ldg(r + 1) - v) - (v - __ldg(r - 1)));
                m = d <= 3.402823466e38f ? fmaxf(m, d) : INFINITY;
            }
            if (y > 0 && y < H - 1) {
                const float d = fabsf((__ldg(r + W) - v) - (v - __ldg(r - W)));
                m = d <= 3.402823466e38f ? fmaxf(m, d) : INFINITY;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&st->ray_bend, __float_as_uint(m));
}

// a / b from r ~ 1 / b: Markstein's correction (IBM J. Res. Dev. 34, 1990) - the remainder a - q b is
// exact in one fused operation. With r within 2^-52 of 1 / b and q within 1.5 x 2^-52 of a / b, both
// relative, q + (a - q b) r is off by 1.5 x 2^-104 before its one rounding, 1.5 x 2^-51 ulp: the result is
// the correctly rounded quotient unless a / b lies within 2^-50 ulp of the middle between two doubles
// (and is then one of the two). Several numerators share one reciprocal.
__device__ __forceinline__ double pm_quot(double a, double b, double r) {
    const double q = __dmul_rn(a, r);
    return __fma_rn(__fma_rn(-q, b, a), r, q);
}

// Geometric term of _pm_cost (_dense.pyx:532-555): mean over the sources with depth maps of
// min(1, |z - d_j| / d_j / geo_tol) at the rounded projection of the window centre.
__device__ __forceinline__ double pm_geo(const PMParams& c, double d, double rpx, double rpy, double rpz) {
    double geo = 0.0;
    if (c.geo_w > 0.0) {
        const double X = c.cr0 + d * rpx, Y = c.cr1 + d * rpy, Z = c.cr2 + d * rpz;
        int ng = 0;
        for (int s = 0; s < c.S; ++s) {
            if (c.dep[s] == nullptr) continue;
            ++ng;
            double e = 1.0, u, v, z;
            if (pm_proj(c.par + 18 * s, X, Y, Z, u, v, z)) {
                const int ui = (int)(u + 0.5), vv = (int)(v + 0.5);
                if (ui >= 0 && vv >= 0 && ui < c.iw[s] && vv < c.ih[s]) {
                    const double dj = __ldg(c.dep[s] + (long long)vv * c.iw[s] + ui);
                    if (isfinite(dj) && dj > 0.0) {
                        e = fabs(z - dj) / dj / c.geo_tol;
                        if (e > 1.0) e = 1.0;
                    }
                }
            }
            geo = geo + e;
        }
        if (ng) geo = geo / (double)ng;
    }
    return geo;
}

// A pixel's window, fixed for one visit.
struct PMPix {
    int y, x;
    int a0, a1, b0, b1;            // offsets inside the image: a0, a0 + step, .. <= a1 (rows), b likewise
    double rpx, rpy, rpz;
    double si, sii;                // sums of I and I^2 over the finite reference values, in window order
    int nfin;
    int slot;                      // the pixel's place in the block (PMCorners)
    float dev;                     // bound of a ray's distance from the corners' bilinear interpolation
    float wmax;                    // largest component of the corner offsets
    bool prune;
};

// Float32 corner offsets (ray_corner - ray_p) of the block's pixels: [corner * 3 + component][pixel].
typedef float PMCorners[12][128];

// One candidate's window sums for M consecutive entries of a source list (uniform over the warp's
// converged lanes): sJ, sJJ, sIJ, and when CHECKED sI, sII and the count of valid samples.
template <int M, bool CHECKED>
__device__ __forceinline__ void pm_sums64(const PMParams& c, const PMPix& px, const int (&src)[M], double num,
                                          const double* n, int& ns, double (&sJ)[M], double (&sJJ)[M], double (&sIJ)[M],
                                          double (&sI)[M], double (&sII)[M], int (&cnt)[M]) {
    const long long HW = (long long)c.H * c.W;
#pragma unroll
    for (int k = 0; k < M; ++k) {
        sJ[k] = 0.0; sJJ[k] = 0.0; sIJ[k] = 0.0; sI[k] = 0.0; sII[k] = 0.0; cnt[k] = 0;
    }
    ns = 0;
    for (int a = px.a0; a <= px.a1; a += c.step) {
        const long long row = (long long)(px.y + a) * c.W + px.x;
        for (int b = px.b0; b <= px.b1; b += c.step) {
            const long long q = row + b;
            const float If = __ldg(c.ref + q);
            if (!(fabsf(If) <= 3.402823466e38f)) continue;
            const double I = If;
            const double qx = __ldg(c.ray + q), qy = __ldg(c.ray + HW + q), qz = __ldg(c.ray + 2 * HW + q);
            const double den = n[0] * qx + n[1] * qy + n[2] * qz;
            if (CHECKED && den >= -1e-9) continue;
            const double t = pm_quot(num, den, rcp_newton(den));
            const double X = c.cr0 + t * qx, Y = c.cr1 + t * qy, Z = c.cr2 + t * qz;
            ++ns;
            const double II = I * I;
#pragma unroll
            for (int k = 0; k < M; ++k) {
                const int s = src[k];
                const double* p = c.par + 18 * s;
                // _proj
                const double dx = X - p[9], dy = Y - p[10], dz = Z - p[11];
                const double xc = p[0] * dx + p[1] * dy + p[2] * dz;
                const double yc = p[3] * dx + p[4] * dy + p[5] * dz;
                const double zc = p[6] * dx + p[7] * dy + p[8] * dz;
                const bool front = !CHECKED || zc > 1e-6;
                const double zq = front ? zc : 1.0;
                const double rz = rcp_newton(zq);
                const double nx = pm_quot(xc, zq, rz), ny = pm_quot(yc, zq, rz);
                // pinhole source: the reference's factor f (1 + r2 (k1 + r2 (k2 + r2 k3)))
                // evaluates to exactly f (r2 >= 0 finite, so every product with 0 is +0)
                double dd = p[12];
                if (!c.pinhole[s]) {
                    const double r2 = nx * nx + ny * ny;
                    dd = p[12] * (1.0 + r2 * (p[13] + r2 * (p[14] + r2 * p[15])));
                }
                const double u = dd * nx + p[16], v = dd * ny + p[17];
                // _bil: floor by an addition rounded toward -inf (the low word of u + 1.5 * 2^52)
                const int iw = c.iw[s], ih = c.ih[s];
                bool in = true;
                double us = u, vs = v;
                if (CHECKED) {   // NaN u / v count as outside
                    in = front && u >= 0.0 && v >= 0.0 && u <= (double)iw - 1.001 && v <= (double)ih - 1.001;
                    us = in ? u : 0.0;
                    vs = in ? v : 0.0;
                }
                const double tu = __dadd_rd(us, 6755399441055744.0), tv = __dadd_rd(vs, 6755399441055744.0);
                int x0 = __double2loint(tu), y0 = __double2loint(tv);
                if (!CHECKED) {
                    // a no-op for the lanes whose window is inside; the others' sums are not used
                    x0 = (int)min((unsigned)x0, (unsigned)(iw - 2));
                    y0 = (int)min((unsigned)y0, (unsigned)(ih - 2));
                }
                const double fx = us - __dsub_rn(tu, 6755399441055744.0), fy = vs - __dsub_rn(tv, 6755399441055744.0);
                MVS_BOUND((long long)y0 * iw + x0 >= 0 && (long long)y0 * iw + x0 + iw + 1 < (long long)iw * ih);
                const float* im = c.img[s] + ((long long)y0 * iw + x0);
                const double a00 = __ldg(im), a01 = __ldg(im + 1), a10 = __ldg(im + iw), a11 = __ldg(im + iw + 1);
                const double J = (a00 * (1.0 - fx) + a01 * fx) * (1.0 - fy) + (a10 * (1.0 - fx) + a11 * fx) * fy;
                if (CHECKED) {
                    const bool ok = in && isfinite(J);
                    sI[k] += ok ? I : 0.0;
                    sJ[k] += ok ? J : 0.0;
                    sII[k] += ok ? II : 0.0;
                    sJJ[k] += ok ? J * J : 0.0;
                    sIJ[k] += ok ? I * J : 0.0;
                    cnt[k] += ok ? 1 : 0;
                } else {
                    sJ[k] += J;
                    sJJ[k] += J * J;
                    sIJ[k] += I * J;
                }
            }
        }
    }
}

// Where the window of plane (d, n) maps to in source s: +1 every sample inside with a margin (and in
// front, and counted), -1 every sample outside, 0 neither shown. The window's rays are within `dev` of
// the bilinear interpolation of its corner rays and the plane's map is projective, so undistorted
// image points lie in the box of the corners' points, widened by the effect of `dev` and of float32
// rounding; a distorted source's factor 1 + r2 (..) is bounded by its terms' absolute values. The bounds
// hold for normals of any length and windows of any size: rounding is in proportion to the map's
// coefficients times the offsets, not to the corners' sums, which cancel where a plane is seen edge-on.
__device__ __forceinline__ int pm_where(const PMParams& c, const PMPix& px, const PMCorners& cor, int s, float num,
                                        float n0, float n1, float n2, float ndr) {
    const float* p = c.parf + 18 * s;
    const float* bs = c.bsf + 3 * s;
    const float rx = (float)px.rpx, ry = (float)px.rpy, rz = (float)px.rpz;
    const float nl = fabsf(n0) + fabsf(n1) + fabsf(n2), den_max = -(1e-4f + 4.f * px.dev) * fmaxf(nl, 1.f);
    float M[3][3], cen[3], bmax = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float b = bs[i], p0 = p[3 * i], p1 = p[3 * i + 1], p2 = p[3 * i + 2];
        M[i][0] = fmaf(b, n0, num * p0);
        M[i][1] = fmaf(b, n1, num * p1);
        M[i][2] = fmaf(b, n2, num * p2);
        cen[i] = fmaf(b, ndr, num * fmaf(p0, rx, fmaf(p1, ry, p2 * rz)));
        bmax = fmaxf(bmax, fabsf(b));
    }
    const float big = bmax * (fabsf(ndr) + nl * px.wmax) +
                      fabsf(num) * (fabsf(rx) + fabsf(ry) + fabsf(rz) + 3.f * px.wmax);
    const float zc = cen[2];                              // camera depth is zc / ndr: < 0 in front
    if (!(zc < -1e-20f)) return 0;
    const float iz = __fdividef(1.0f, zc);
    float xlo = INFINITY, xhi = -INFINITY, ylo = INFINITY, yhi = -INFINITY;
    bool good = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float w0 = cor[3 * k][px.slot], w1 = cor[3 * k + 1][px.slot], w2 = cor[3 * k + 2][px.slot];
        const float v0 = fmaf(M[0][0], w0, fmaf(M[0][1], w1, fmaf(M[0][2], w2, cen[0])));
        const float v1 = fmaf(M[1][0], w0, fmaf(M[1][1], w1, fmaf(M[1][2], w2, cen[1])));
        const float v2 = fmaf(M[2][0], w0, fmaf(M[2][1], w1, fmaf(M[2][2], w2, cen[2])));
        const float den = fmaf(n0, w0, fmaf(n1, w1, fmaf(n2, w2, ndr)));
        good = good && den < den_max && v2 < 1e-2f * den && v2 < 0.5f * zc;
        const float r = __fdividef(1.0f, v2);
        xlo = fminf(xlo, v0 * r);
        xhi = fmaxf(xhi, v0 * r);
        ylo = fminf(ylo, v1 * r);
        yhi = fmaxf(yhi, v1 * r);
    }
    const float ax = fmaxf(fabsf(xlo), fabsf(xhi)), ay = fmaxf(fabsf(ylo), fabsf(yhi));
    // errors of the box, in image units of the undistorted plane: `dev` through the map (its change
    // over the window is at most 2 x, by v2 < zc / 2), float32 rounding of the composed map
    const float m2 = fabsf(M[2][0]) + fabsf(M[2][1]) + fabsf(M[2][2]);
    const float m0 = fabsf(M[0][0]) + fabsf(M[0][1]) + fabsf(M[0][2]), m1 = fabsf(M[1][0]) + fabsf(M[1][1]) + fabsf(M[1][2]);
    const float ex = -iz * (4.f * (m0 + ax * m2) * px.dev + 4e-6f * big * (1.f + ax));
    const float ey = -iz * (4.f * (m1 + ay * m2) * px.dev + 4e-6f * big * (1.f + ay));
    const float f = p[12], cx = p[16], cy = p[17];
    float sd = 0.f;
    if (!c.pinhole[s]) {
        const float r2 = (ax + ex) * (ax + ex) + (ay + ey) * (ay + ey);
        sd = 1.001f * r2 * (fabsf(p[13]) + r2 * (fabsf(p[14]) + r2 * fabsf(p[15])));
    }
    good = good && sd < 0.5f && f > 0.f && ex * f < 8.f && ey * f < 8.f;
    xlo -= ex; xhi += ex; ylo -= ey; yhi += ey;
    const float ulo = fmaf(f, xlo * (xlo < 0.f ? 1.f + sd : 1.f - sd), cx), uhi = fmaf(f, xhi * (xhi > 0.f ? 1.f + sd : 1.f - sd), cx);
    const float vlo = fmaf(f, ylo * (ylo < 0.f ? 1.f + sd : 1.f - sd), cy), vhi = fmaf(f, yhi * (yhi > 0.f ? 1.f + sd : 1.f - sd), cy);
    const float w = (float)c.iw[s], h = (float)c.ih[s];
    const float m = 0.5f + 2e-5f * (f + fabsf(cx) + fabsf(cy) + w + h);
    if (!good) return 0;                                  // NaN anywhere above fails a test
    if (uhi < -m || vhi < -m || ulo > w + m || vlo > h + m) return -1;
    return ulo > m && vlo > m && uhi < w - 1.001f - m && vhi < h - 1.001f - m ? 1 : 0;
}

// NCC of one source from its window sums (_dense.pyx:505-528).
__device__ __forceinline__ double pm_ncc64(int ns, int cnt, double sI, double sJ, double sII, double sJJ, double sIJ) {
    if (ns < 4 || (double)cnt < 0.7 * (double)ns) return -1.0;
    const double dc = (double)cnt;
    const double mi = sI / dc, mj = sJ / dc;
    const double vi = sII / dc - mi * mi;
    const double vj = sJJ / dc - mj * mj;
    const double cv = sIJ / dc - mi * mj;
    return (vi < 1e-8 || vj < 1e-8) ? 0.0 : cv / sqrt(vi * vj);
}

template <int M>
__device__ __forceinline__ void pm_batch64(const PMParams& c, const PMPix& px, unsigned group, bool checked,
                                           unsigned in, unsigned out, double num, const double* n, double* ncc) {
    int src[M];
#pragma unroll
    for (int k = 0; k < M; ++k) {
        src[k] = __ffs(group) - 1;
        group &= group - 1;
    }
    double sJ[M], sJJ[M], sIJ[M], sI[M], sII[M];
    int ns, cnt[M];
    bool redo = checked;
    if (!checked) {
        pm_sums64<M, false>(c, px, src, num, n, ns, sJ, sJJ, sIJ, sI, sII, cnt);
        // a non-finite source value in the window poisons the sums
#pragma unroll
        for (int k = 0; k < M; ++k) redo = redo || (((in >> src[k]) & 1u) && !isfinite(sJJ[k]));
        ns = px.nfin;
#pragma unroll
        for (int k = 0; k < M; ++k) {
            sI[k] = px.si;
            sII[k] = px.sii;
            cnt[k] = px.nfin;
        }
    }
    if (redo) pm_sums64<M, true>(c, px, src, num, n, ns, sJ, sJJ, sIJ, sI, sII, cnt);
#pragma unroll
    for (int k = 0; k < M; ++k)
        ncc[src[k]] = !checked && ((out >> src[k]) & 1u) ? -1.0 : pm_ncc64(ns, cnt[k], sI[k], sJ[k], sII[k], sJJ[k], sIJ[k]);
}

// The cost of plane (d, n), or +inf where it provably is not below `best` (a candidate that the
// caller then does not accept). best = +inf: always evaluated.
__device__ double pm_cost(const PMParams& c, const PMPix& px, const PMCorners& cor, double d, const double* n, double best,
                          double& ncc_out) {
    const double ndr = n[0] * px.rpx + n[1] * px.rpy + n[2] * px.rpz;
    if (ndr >= -1e-6 || d <= 0.0) {
        ncc_out = 0.0;   // unused by the caller for cost 10 (never accepted over a real cost)
        return 10.0;
    }
    const double gterm = c.geo_w * pm_geo(c, d, px.rpx, px.rpy, px.rpz);
    // PM_PRUNE: the NCC of values up to 6 in magnitude exceeds 1 by less than 1e-3 through rounding
    // (window sums of at most 400 samples carry < 1e-12; the variances are at least 1e-8), so the cost
    // is at least gterm - 1e-3
    if (px.prune && gterm - 1e-3 >= best) {
        ncc_out = 0.0;
        return __longlong_as_double(0x7ff0000000000000LL);
    }
    const double num = d * ndr;
    const unsigned all = (1u << c.S) - 1u;
    unsigned in = 0, out = 0;
    for (int s = 0; s < c.S; ++s) {
        const int w = pm_where(c, px, cor, s, (float)num, (float)n[0], (float)n[1], (float)n[2], (float)ndr);
        in |= w > 0 ? 1u << s : 0u;
        out |= w < 0 ? 1u << s : 0u;
    }
    double ncc[MVS_MAX_SOURCES];
    for (int s = 0; s < c.S; ++s) ncc[s] = -1.0;
    // the converged lanes walk the same source lists: the sources inside (or outside) for every lane
    // without tests, then those that some lane has to test
    const unsigned lanes = __activemask();
    const unsigned need = __reduce_or_sync(lanes, all & ~out), test = __reduce_or_sync(lanes, all & ~out & ~in);
    for (int checked = 0; checked < 2; ++checked) {
        unsigned list = checked ? need & test : need & ~test;
        while (list) {
            const int m = min(__popc(list), PM_PASS);
            unsigned group = 0;
            for (int k = 0; k < m; ++k) {
                group |= list & (0u - list);
                list &= list - 1;
            }
            if (m == 2) pm_batch64<2>(c, px, group, checked, in, out, num, n, ncc);
            else pm_batch64<1>(c, px, group, checked, in, out, num, n, ncc);
        }
    }
    // descending insertion sort (S <= 16), then the mean of the first top_k
    for (int a = 1; a < c.S; ++a) {
        const double tmp = ncc[a];
        int b = a - 1;
        while (b >= 0 && ncc[b] < tmp) {
            ncc[b + 1] = ncc[b];
            --b;
        }
        ncc[b + 1] = tmp;
    }
    const int kk = c.top_k < c.S ? c.top_k : c.S;
    double photo = 0.0;
    for (int a = 0; a < kk; ++a) photo = photo + ncc[a];
    photo = photo / (double)kk;
    ncc_out = photo;
    return (1.0 - photo) + gterm;
}

// Resident blocks of 128 threads per SM, 2 sources a pass (4 sources a pass spilled: 11.5 against 8.0 ms
// with one thread walking a pixel's candidates). All of a call's launches with a lane per candidate, ms,
// at 4 / 5 / 6 / 8 blocks (128 / 96 / 80 / 64 registers): a 1600 x 1200 repair (4 sources, 5 x 5 samples, a
// third of the pixels active, geometric term) 6.07 / 6.23 / 6.27 / 5.84, 5 views of 800 x 600 15.7 / 16.6 /
// 17.4 / 17.9, 2000 x 1500 with 8 sources, 7 x 7 samples and every pixel active 117.5 / 119.6 / 117.8 /
// 116.3, 320 x 240 1.62 / 1.78 / 1.85 / 1.91: within 2 % on large views, where fewer registers pay for more
// warps, and fewer blocks better by up to 9 % on small ones, whose pixels do not fill the chip; 5 lies
// between. One thread per pixel, all windows and tests, three divisions a sample: 36.0 and 54.2 on the first two.
constexpr int PM_MIN_BLOCKS = 5;

// Pixel of pass number t (raster order of the colour's pixels): false past the image.
__device__ __forceinline__ bool pm_pixel(const PMParams& c, long long t, int& y, int& x) {
    const int half_w = (c.W + 1) / 2;
    if (t >= (long long)c.H * half_w) return false;
    y = (int)(t / half_w);
    x = 2 * (int)(t - (long long)y * half_w) + ((y + c.colour) & 1);
    return x < c.W;
}

// The two random trials of _dense.pyx:646-663 in the order of the reference: 4 draws per trial
// (depth, then the three normal components), all 8 drawn even when a trial is skipped.
template <typename CostFn>
__device__ __forceinline__ void pm_trials(const PMParams& c, unsigned st, float& dcur, float* ncur, double& best,
                                          double& sc, unsigned long long& changed, CostFn&& cost) {
#pragma unroll 1
    for (int tr = 0; tr < 2; ++tr) {
        const double u0 = xs_draw(st);
        const double u1 = xs_draw(st);
        const double u2 = xs_draw(st);
        const double u3 = xs_draw(st);
        const double dp = (double)dcur * (1.0 + c.dd_scale * (2.0 * u0 - 1.0));
        double nb[3];
        nb[0] = (double)ncur[0] + c.nn_scale * (2.0 * u1 - 1.0);
        nb[1] = (double)ncur[1] + c.nn_scale * (2.0 * u2 - 1.0);
        nb[2] = (double)ncur[2] + c.nn_scale * (2.0 * u3 - 1.0);
        const double nn = sqrt(nb[0] * nb[0] + nb[1] * nb[1] + nb[2] * nb[2]);
        if (nn < 1e-9 || dp < c.dmin || dp > c.dmax) continue;
        nb[0] = nb[0] / nn;
        nb[1] = nb[1] / nn;
        nb[2] = nb[2] / nn;
        double ph;
        const double cst = cost(dp, nb, best, ph);
        if (cst < best) {
            best = cst;
            sc = ph;
            dcur = (float)dp;
            ncur[0] = (float)nb[0];
            ncur[1] = (float)nb[1];
            ncur[2] = (float)nb[2];
            ++changed;
        }
    }
}

// End of a pixel's visit: score, cost cache, change count (depth / normal written by the caller).
__device__ __forceinline__ void pm_finish(const PMParams& c, long long idx, float dcur, double best, double sc,
                                          unsigned long long changed) {
    if (c.cost_cache) {
        const bool keep = changed == 0 && isfinite(dcur);
        c.cost_cache[idx] = keep ? best : __longlong_as_double(0x7ff8000000000000LL);
        if (keep) c.score_cache[idx] = sc;
    }
    c.score[idx] = (float)sc;
    if (changed && c.changed) atomicAdd(c.changed, changed);
}

// PHASE 0: the cost of the current plane where the previous visit did not leave it; PHASE 1: the random
// trials (both one thread per active pixel); PHASE 2: propagation, 8 lanes per active pixel, one
// candidate each - the neighbours' planes do not change during a pass, so the candidates' costs are
// independent, and every lane then takes the decisions in the reference's order from the shared
// costs. (A thread walking its 8 candidates left SMs idle behind the longest threads - 8 % of the warps
// active on average at 800 x 600, whose active pixels are one round of blocks: 1600 x 1200 repair 6.6
// -> 4.6 ms for phases 0 and 2, 5 views of 800 x 600 19.9 -> 11.5 ms.)
enum { PM_CURRENT = 0, PM_TRIALS = 1, PM_PROPAGATE = 2 };
template <int PHASE>
__global__ void __launch_bounds__(128, PM_MIN_BLOCKS) pm_kernel(const __grid_constant__ PMParams c) {
    __shared__ PMCorners cor;
    constexpr int LANES = PHASE == PM_PROPAGATE ? 8 : 1;
    const unsigned slot = blockIdx.x * (128u / LANES) + threadIdx.x / LANES;
    if (slot >= *c.n_list) return;
    const long long t = c.list[slot];
    PMPix px;
    px.slot = threadIdx.x / LANES;
    if (!pm_pixel(c, t, px.y, px.x)) return;          // (list entries are pixels)
    const int y = px.y, x = px.x;
    const long long HW = (long long)c.H * c.W, idx = (long long)y * c.W + x;
    unsigned flag = 0;
    if (PHASE == PM_TRIALS) {
        flag = c.flags[t];
        if (!(flag & 1u)) {                           // no draws: the visit ends with propagation's result
            pm_finish(c, idx, c.depth[idx], c.pbest[t], c.psc[t], flag >> 1);
            return;
        }
    }
    float dcur = c.depth[idx];
    float ncur[3] = {c.normal[idx], c.normal[HW + idx], c.normal[2 * HW + idx]};
    double best, sc, ncc;
    if (PHASE == PM_CURRENT) {
        // reused from the previous visit when that visit kept the plane it started with (the cost was
        // then computed from these very float32 values)
        const double cached = c.cost_cache ? c.cost_cache[idx] : __longlong_as_double(0x7ff8000000000000LL);
        if (!isfinite(dcur) || cached == cached) {
            c.pbest[t] = isfinite(dcur) ? cached : 1e9;
            c.psc[t] = isfinite(dcur) ? c.score_cache[idx] : -1.0;
            return;
        }
    }
    {
        // the window clipped to the image, its corner rays and its reference sums
        // (the first offset inside the image lies within a step of it; its parts may pass 2^31)
        const int r = c.r, st = c.step;
        px.a0 = y < r ? (int)(((unsigned)(r - y - 1) / st + 1u) * st - r) : -r;
        px.b0 = x < r ? (int)(((unsigned)(r - x - 1) / st + 1u) * st - r) : -r;
        px.a1 = min(c.last, c.H - 1 - y);
        px.b1 = min(c.last, c.W - 1 - x);
        const float rx = __ldg(c.ray + idx), ry = __ldg(c.ray + HW + idx), rz = __ldg(c.ray + 2 * HW + idx);
        px.rpx = rx; px.rpy = ry; px.rpz = rz;
        float wmax = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int yy = k < 2 ? max(y - r, 0) : y + min(r, c.H - 1 - y), xx = (k & 1) ? x + min(r, c.W - 1 - x) : max(x - r, 0);
            const long long q = (long long)yy * c.W + xx;
            const float w0 = __ldg(c.ray + q) - rx, w1 = __ldg(c.ray + HW + q) - ry, w2 = __ldg(c.ray + 2 * HW + q) - rz;
            cor[3 * k][px.slot] = w0;
            cor[3 * k + 1][px.slot] = w1;
            cor[3 * k + 2][px.slot] = w2;
            wmax = fmaxf(wmax, fmaxf(fabsf(w0), fmaxf(fabsf(w1), fabsf(w2))));
        }
        px.wmax = wmax;
        px.si = px.sii = 0.0;
        px.nfin = 0;
        for (int a = px.a0; a <= px.a1; a += st)
            for (int b = px.b0; b <= px.b1; b += st) {
                const float If = __ldg(c.ref + (long long)(y + a) * c.W + x + b);
                if (!(fabsf(If) <= 3.402823466e38f)) continue;
                const double I = If;
                px.si += I;
                px.sii += I * I;
                ++px.nfin;
            }
        // piecewise linear interpolation between points 2 r apart is off by at most r^2 / 2 second
        // differences per direction
        px.dev = c.r2 * __uint_as_float(c.stats->ray_bend);
        px.prune = __uint_as_float(c.stats->max_abs) <= 6.f && c.few;
    }
    auto cost = [&](double d, const double* nb, double bound, double& ph) { return pm_cost(c, px, cor, d, nb, bound, ph); };
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    if (PHASE == PM_CURRENT) {
        const double n[3] = {ncur[0], ncur[1], ncur[2]};
        c.pbest[t] = cost((double)dcur, n, inf, ncc);
        c.psc[t] = ncc;
        return;
    }
    best = c.pbest[t];
    sc = c.psc[t];
    unsigned long long changed = 0;
    if (PHASE == PM_TRIALS) {
        changed = flag >> 1;
        pm_trials(c, c.pstate[t], dcur, ncur, best, sc, changed, cost);
        c.depth[idx] = dcur;
        c.normal[idx] = ncur[0];
        c.normal[HW + idx] = ncur[1];
        c.normal[2 * HW + idx] = ncur[2];
        pm_finish(c, idx, dcur, best, sc, changed);
        return;
    }
    const int lane = threadIdx.x & 7;
    const unsigned gmask = 0xffu << (threadIdx.x & 24);
    // offsets (-1, 0), (1, 0), (0, -1), (0, 1), then the same by 5
    const int reach = lane < 4 ? 1 : 5, side = (lane & 1) ? reach : -reach;
    const int yn = y + ((lane & 2) ? 0 : side), xn = x + ((lane & 2) ? side : 0);
    double cst = inf;
    ncc = 0.0;
    float dp_f = 0.f, n0 = 0.f, n1 = 0.f, n2 = 0.f;
    if (yn >= 0 && xn >= 0 && yn < c.H && xn < c.W) {
        const long long nidx = (long long)yn * c.W + xn;
        const float dnb = c.depth[nidx];
        n0 = c.normal[nidx];
        n1 = c.normal[HW + nidx];
        n2 = c.normal[2 * HW + nidx];
        const double nb[3] = {n0, n1, n2};
        const double dn = nb[0] * __ldg(c.ray + nidx) + nb[1] * __ldg(c.ray + HW + nidx) + nb[2] * __ldg(c.ray + 2 * HW + nidx);
        const double ndr = nb[0] * px.rpx + nb[1] * px.rpy + nb[2] * px.rpz;
        const double dp = (double)dnb * dn / ndr;
        if (isfinite(dnb) && !(ndr >= -1e-6) && !(dp < c.dmin || dp > c.dmax)) {
            cst = cost(dp, nb, best, ncc);
            dp_f = (float)dp;
        }
    }
    __syncwarp(gmask);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const double ck = __shfl_sync(gmask, cst, k, 8), pk = __shfl_sync(gmask, ncc, k, 8);
        const float dk = __shfl_sync(gmask, dp_f, k, 8), a0 = __shfl_sync(gmask, n0, k, 8);
        const float a1 = __shfl_sync(gmask, n1, k, 8), a2 = __shfl_sync(gmask, n2, k, 8);
        if (ck < best) {
            best = ck;
            sc = pk;
            dcur = dk;
            ncur[0] = a0; ncur[1] = a1; ncur[2] = a2;
            ++changed;
        }
    }
    if (lane != 0) return;
    if (changed) {
        c.depth[idx] = dcur;
        c.normal[idx] = ncur[0];
        c.normal[HW + idx] = ncur[1];
        c.normal[2 * HW + idx] = ncur[2];
    }
    c.pbest[t] = best;
    c.psc[t] = sc;
    c.flags[t] = (unsigned char)((isfinite(dcur) ? 1u : 0u) | ((unsigned)changed << 1));
}

// ---------------------------------------------------------------- draw offsets of a colour pass

constexpr int PM_SCAN_BLOCK = 1024;

// Exclusive prefix sum over a block of PM_SCAN_BLOCK (32 warps) threads; `total` = the block's
// sum. Called once per kernel (its shared words are not reused).
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned& total) {
    __shared__ unsigned warp_off[32];
    __shared__ unsigned tot_s;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) warp_off[w] = inc;
    __syncthreads();
    if (w == 0) {
        const unsigned wt = warp_off[lane];
        unsigned wi = wt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += u;
        }
        warp_off[lane] = wi - wt;
        if (lane == 31) tot_s = wi;
    }
    __syncthreads();
    total = tot_s;
    return warp_off[w] + inc - v;
}

// Drawing pixels per block of PM_SCAN_BLOCK pass pixels.
__global__ void __launch_bounds__(PM_SCAN_BLOCK) pm_count_kernel(const unsigned char* flags, long long n,
                                                                  unsigned* bsum) {
    const long long t = (long long)blockIdx.x * PM_SCAN_BLOCK + threadIdx.x;
    const int f = t < n ? (flags[t] & 1) : 0;
    const int cnt = __syncthreads_count(f);
    if (threadIdx.x == 0) bsum[blockIdx.x] = (unsigned)cnt;
}

// One block: block counts -> exclusive block offsets (in place); the stream state after the
// pass's 8 * total draws goes to rng[nxt].
__global__ void __launch_bounds__(PM_SCAN_BLOCK) pm_scan_kernel(unsigned* bsum, int nb, unsigned* rng, int cur,
                                                                 int nxt, const __grid_constant__ PMJump J) {
    const int per = (nb + PM_SCAN_BLOCK - 1) / PM_SCAN_BLOCK;
    const int beg = min(nb, (int)threadIdx.x * per), end = min(nb, beg + per);
    unsigned s = 0;
    for (int i = beg; i < end; ++i) s += bsum[i];
    unsigned total = 0;
    unsigned run = block_exclusive_scan(s, total);
    for (int i = beg; i < end; ++i) {
        const unsigned v = bsum[i];
        bsum[i] = run;
        run += v;
    }
    if (threadIdx.x == 0) rng[nxt] = jump8(J, rng[cur], total);
}

// Per drawing pixel: the stream state before its first draw (0 for pixels that do not draw; a
// xorshift32 state is never 0). The jump of a pixel splits into the jump to its warp's first draw, which
// the lanes of the first warp form for all 32 warps at once, and at most 31 pixels within the warp,
// from nibble tables in shared memory (8 words read per matrix product instead of 32 masks and
// xors): every pixel jumping by its block-wide number took 388 us a pass at 4000 x 3000.
__global__ void __launch_bounds__(PM_SCAN_BLOCK) pm_state_kernel(const unsigned char* flags, long long n,
                                                                  const unsigned* boff, const unsigned* rng, int cur,
                                                                  const __grid_constant__ PMJump J, unsigned* pstate) {
    __shared__ unsigned tab[5][8][16];      // t[j] applied to nibble q of a state
    __shared__ unsigned wcount[32], wbase[32];
    __shared__ unsigned base;
    const long long t = (long long)blockIdx.x * PM_SCAN_BLOCK + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool f = t < n && (flags[t] & 1u);
    const unsigned draw = __ballot_sync(0xffffffffu, f);
    if (lane == 0) wcount[w] = __popc(draw);
    if (threadIdx.x < 5 * 8 * 16) {
        const int j = threadIdx.x / 128, q = (threadIdx.x / 16) % 8, v = threadIdx.x % 16;
        unsigned r = 0;
        for (int b = 0; b < 4; ++b)
            if (v & (1 << b)) r ^= J.t[j].col[4 * q + b];
        tab[j][q][v] = r;
    }
    if (threadIdx.x == PM_SCAN_BLOCK - 1) base = jump8(J, rng[cur], boff[blockIdx.x]);
    __syncthreads();
    if (w == 0) {                           // exclusive prefix of the warps' draws, and their states
        unsigned inc = wcount[lane];
        const unsigned own = inc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        wbase[lane] = jump8(J, base, inc - own);
    }
    __syncthreads();
    if (t >= n) return;
    unsigned s = wbase[w];
    const unsigned k = __popc(draw & ((1u << lane) - 1u));
#pragma unroll
    for (int j = 0; j < 5; ++j)
        if (k & (1u << j)) {
            unsigned r = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) r ^= tab[j][q][(s >> (4 * q)) & 15u];
            s = r;
        }
    pstate[t] = f ? s : 0u;
}

// The active pixels of a colour: per block of PM_SCAN_BLOCK pass pixels their number, and (after
// pm_offsets_kernel) their pass pixel numbers in raster order.
__device__ __forceinline__ bool pm_is_active(const unsigned char* active, int H, int W, int colour, long long t) {
    const int half_w = (W + 1) / 2;
    if (t >= (long long)H * half_w) return false;
    const int y = (int)(t / half_w), x = 2 * (int)(t - (long long)y * half_w) + ((y + colour) & 1);
    return x < W && active[(long long)y * W + x];
}
__global__ void __launch_bounds__(PM_SCAN_BLOCK) pm_active_count_kernel(const unsigned char* active, int H, int W,
                                                                        int colour, unsigned* bsum) {
    const long long t = (long long)blockIdx.x * PM_SCAN_BLOCK + threadIdx.x;
    const int cnt = __syncthreads_count(pm_is_active(active, H, W, colour, t));
    if (threadIdx.x == 0) bsum[blockIdx.x] = (unsigned)cnt;
}
// One block: counts -> exclusive offsets in place, and their total.
__global__ void __launch_bounds__(PM_SCAN_BLOCK) pm_offsets_kernel(unsigned* bsum, int nb, unsigned* total_out) {
    const int per = (nb + PM_SCAN_BLOCK - 1) / PM_SCAN_BLOCK;
    const int beg = min(nb, (int)threadIdx.x * per), end = min(nb, beg + per);
    unsigned s = 0;
    for (int i = beg; i < end; ++i) s += bsum[i];
    unsigned total = 0;
    unsigned run = block_exclusive_scan(s, total);
    for (int i = beg; i < end; ++i) {
        const unsigned v = bsum[i];
        bsum[i] = run;
        run += v;
    }
    if (threadIdx.x == 0) *total_out = total;
}
__global__ void __launch_bounds__(PM_SCAN_BLOCK) pm_active_list_kernel(const unsigned char* active, int H, int W,
                                                                       int colour, const unsigned* boff,
                                                                       unsigned* list) {
    const long long t = (long long)blockIdx.x * PM_SCAN_BLOCK + threadIdx.x;
    const bool f = pm_is_active(active, H, W, colour, t);
    unsigned total;
    const unsigned excl = block_exclusive_scan(f ? 1u : 0u, total);
    if (f) list[boff[blockIdx.x] + excl] = (unsigned)t;
}

__global__ void pm_rng_init_kernel(unsigned* rng, const unsigned* from, unsigned seed) {
    rng[0] = from ? *from : seed;
}

// The 2 x 2 bilinear footprints of a source image (PMParams::quad). The last row and column, which
// are never a footprint's top-left tap (every tap offset is clamped to (h - 2) w + w - 2), repeat
// the edge.
__global__ void __launch_bounds__(256) pm_quad_kernel(const float* __restrict__ im, int w, int h,
                                                      float4* __restrict__ quad) {
    const long long n = (long long)w * h;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int y = (int)(i / w), x = (int)(i - (long long)y * w);
        const long long r0 = (long long)y * w, r1 = (long long)min(y + 1, h - 1) * w;
        const int x1 = min(x + 1, w - 1);
        quad[i] = make_float4(__ldg(im + r0 + x), __ldg(im + r1 + x), __ldg(im + r0 + x1), __ldg(im + r1 + x1));
    }
}

// ---------------------------------------------------------------- float32 evaluation (MVS_PM_FP32)
//
// The same visits, candidates, draws and acceptance rule as pm_kernel, with the window costs
// evaluated in float32 and the work of one pixel spread over a group of L lanes, one per source:
//
//   * geometry: for a plane (d, n) and a pinhole source s, the camera point of window sample q is
//     M_s ray_q / (n . ray_q) with M_s = b_s n^T + d (n . ray_p) R_s and b_s = R_s (C_ref - C_s)
//     (the reference's ray-plane intersection followed by _proj, multiplied through by
//     n . ray_q). Per (candidate, source) M_s is composed in float64, folded with f, cx, cy and an
//     integer source anchor (U0, V0) at the window centre, and rounded once; per sample only
//     ray_q - ray_p enters, in float32, so source positions carry ~1e-6 px of rounding error;
//   * validity: when the four corners of the (clipped) window map inside the source with a 1 px
//     margin and in front of it, every sample does (a projective map keeps the window inside the
//     convex hull of its corner images) and the per-sample tests are skipped; otherwise each
//     sample is tested as in the reference (camera depth > 1e-6, 0 <= u <= w - 1.001, ...);
//   * sums: reference values are shifted by the window mean of the reference and source values
//     by the source's value at the window centre, so the float32 variance terms do not cancel;
//   * the lanes of a pixel sort their NCCs with a shuffle network (top-k mean) and sum the
//     geometric term; every lane follows the same candidate sequence and decision.
// Float32 costs differ from the float64 ones by ~1e-7 (measured 99.9th percentile 2e-6), so the
// strict '<' can decide near-ties differently; the float64 mode decides them as the reference does.

// Resident blocks of 256 threads per SM for the lane kernel (propagation; trials). Propagation of 4
// iterations at 4000 x 3000, 8 sources, 7 x 7: 252 ms with single samples at 5 blocks (48 registers), in
// pairs of a row 239 ms at 5, 232 ms at 4 (64 registers), 248 ms at 3, in pairs of the whole window and
// with a shorter unit set-up 217 ms at 4. What bounds it is latency at that occupancy: 60 % of the issue
// slots are used (~130 of the 217 ms), stalls are led by the footprint loads.
constexpr int PM_LANE_MIN_BLOCKS = 4;

__device__ __forceinline__ int pmf_floor(float x, float& f) {   // |x| < 2^22
    const float t = __fadd_rd(x, 12582912.0f);
    f = __fsub_rn(t, 12582912.0f);
    return __float_as_int(t) - 0x4B400000;
}

// The same floor, returning the raw bits of x + 1.5 * 2^23 (floor(x) + 0x4B400000).
__device__ __forceinline__ unsigned pmf_floor_bits(float x, float& f) {   // |x| < 2^22
    const float t = __fadd_rd(x, 12582912.0f);
    f = __fsub_rn(t, 12582912.0f);
    return (unsigned)__float_as_int(t);
}

__device__ __forceinline__ float2 pm_dup(float x) { return make_float2(x, x); }
// a - b elementwise with one rounding (b (-1) + a)
__device__ __forceinline__ float2 pm_sub2(float2 a, float2 b) { return __ffma2_rn(b, pm_dup(-1.0f), a); }
// The hardware's approximation of 1 / x for normal x (the bits of __fdividef(1, x) there)
__device__ __forceinline__ float pm_rcp_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The smaller (larger) of a and b, NaN when either is.
__device__ __forceinline__ float pm_min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float pm_max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// A pixel's window as the cost code reads it: sample (row, k) = e-th of the window as
// (ray_q - ray_p, I_q - mI) with I = NaN where there is no sample (outside the image or a
// non-finite reference value), and the ray offsets of the clipped window's four corners. PAIRS:
// neighbouring samples come as packed pairs of each component, for the packed arithmetic of
// pm_window_sums: samples e and e + 1 of the whole window (FLAT: only the last pair of an odd window
// has a surplus second sample), or of a row (then every row of an odd side has one).
//   PMWinStaged: staged once per visit in shared memory by the pixel's lane group;
//   PMWinPairs:  the same for a side known at compile time, pair by pair (32 bytes: x x y y z z I I);
//   PMWinTile:   read from the warp's shared tile of raw rays and reference values (one lane per
//                pixel; one plane per component, so that a pair of columns is one 8-byte load and the
//                lanes' loads are contiguous), the offsets formed on each read - the same float32
//                operations, so the same values (positions outside the image hold masked samples
//                either way). PAIRS at step 1, where a lane's columns start on an even one.
struct PMWinStaged {
    static constexpr bool PAIRS = false, FLAT = false;
    const float4* w;      // NW samples, then the 4 corners
    __device__ __forceinline__ float4 at(int, int, int e) const { return w[e]; }
    __device__ __forceinline__ float4 corner(int k4, int nw) const { return w[nw + k4]; }
};
template <int NSIDE>
struct PMWinPairs {
    static constexpr bool PAIRS = true, FLAT = true;
    static constexpr int NW = NSIDE * NSIDE, NP = (NW + 1) / 2;   // samples, pairs
    const float4* w;
    static __device__ __forceinline__ int slot(int e) { return (e >> 1) * 8 + (e & 1); }
    __device__ __forceinline__ float4 at(int, int, int e) const {
        const float* f = reinterpret_cast<const float*>(w) + slot(e);
        return make_float4(f[0], f[2], f[4], f[6]);
    }
    __device__ __forceinline__ float4 corner(int k4, int) const { return w[2 * NP + k4]; }
    __device__ __forceinline__ void pair(int, int m, float2& x, float2& y, float2& z, float2& i) const {
        const float4 a = w[2 * m], b = w[2 * m + 1];
        x = make_float2(a.x, a.y);
        y = make_float2(a.z, a.w);
        z = make_float2(b.x, b.y);
        i = make_float2(b.z, b.w);
    }
};
template <bool STEP1>
struct PMWinTile {
    static constexpr bool PAIRS = STEP1, FLAT = false;
    const float* t;       // x plane at the window's first sample (row y - r, column x - r)
    int plane;            // entries of one plane (x, y, z, I)
    int rs, cs;           // tile offsets of one window row and one window column
    int cy0, cy1, cx0, cx1;   // tile offsets of the clipped corners' rows and columns
    float rpx, rpy, rpz, mI;
    __device__ __forceinline__ float4 at(int row, int k, int) const {
        const float* v = t + row * rs + k * cs;
        return make_float4(v[0] - rpx, v[plane] - rpy, v[2 * plane] - rpz, v[3 * plane] - mI);
    }
    __device__ __forceinline__ float4 corner(int k4, int) const {
        const float* v = t + (k4 < 2 ? cy0 : cy1) + ((k4 & 1) ? cx1 : cx0);
        return make_float4(v[0] - rpx, v[plane] - rpy, v[2 * plane] - rpz, 0.f);
    }
    __device__ __forceinline__ void pair(int row, int m, float2& x, float2& y, float2& z, float2& i) const {
        const float* v = t + row * rs + 2 * m;
        x = pm_sub2(*reinterpret_cast<const float2*>(v), pm_dup(rpx));
        y = pm_sub2(*reinterpret_cast<const float2*>(v + plane), pm_dup(rpy));
        z = pm_sub2(*reinterpret_cast<const float2*>(v + 2 * plane), pm_dup(rpz));
        i = pm_sub2(*reinterpret_cast<const float2*>(v + 3 * plane), pm_dup(mI));
    }
};

// Window statistics of a pixel, fixed for one visit.
template <class Acc>
struct PMWinT {
    Acc acc;
    int side, nw;         // samples along a side, in the window
    float nfin;           // samples with a finite reference value inside the image
    float si, sii;        // sum of (I - mI) and (I - mI)^2 over those samples
    bool allfin;          // every sample has a finite reference value inside the image
};

// Pairs of a flat window in flight (24 full pairs at 7 x 7, 12 at 5 x 5); propagation of 4 iterations at
// 4000 x 3000, 8 sources: 2 / 3 / 4 pairs 223.0 / 216.7 / 223.6 ms; row by row (28 pairs, 4 in
// flight) 232 ms.
constexpr int PM_FLAT_AHEAD = 3;

// One source's window sums. CHECKED: every sample tested as in the reference (camera depth,
// source bounds, finite value) and the reference sums formed per source; otherwise (the whole
// window maps inside the source, no sample near a test) only the three source sums are formed.
// ALLFIN: no reference sample is missing (no masking of the reference terms).
template <int NSIDE, bool CHECKED, bool ALLFIN, class Acc>
__device__ __forceinline__ void pm_window_sums(const Acc& win, int side_rt, const float* A, const float* B,
                                               const float* C, float a0, float b0, float c0, float n0, float n1,
                                               float n2, float denp, float lou, float hiu, float lov, float hiv,
                                               unsigned kb, const float4* qd, int sw, unsigned last,
                                               float mJ,
                                               float& T1, float& T2, float& X, float& S1, float& S2, float& cnt,
                                               float& ns) {
    if constexpr (Acc::PAIRS && NSIDE > 0 && !CHECKED) {
        // two samples at a time in packed float32 (each element rounds as its scalar operation, the
        // sums still run sample by sample): coordinates, floors and fractions pair up over the
        // samples, the interpolation along x over a footprint's two rows
        const float2 A0 = pm_dup(A[0]), A1 = pm_dup(A[1]), A2 = pm_dup(A[2]), a0p = pm_dup(a0);
        const float2 B0 = pm_dup(B[0]), B1 = pm_dup(B[1]), B2 = pm_dup(B[2]), b0p = pm_dup(b0);
        const float2 C0 = pm_dup(C[0]), C1 = pm_dup(C[1]), C2 = pm_dup(C[2]), c0p = pm_dup(c0);
        const float2 bias = pm_dup(12582912.0f), nbias = pm_dup(-12582912.0f);
        auto two = [&](int row, int m, bool both) {
            float2 x, y, z, iv;
            win.pair(row, m, x, y, z, iv);
            const float2 cq = __ffma2_rn(C0, x, __ffma2_rn(C1, y, __ffma2_rn(C2, z, c0p)));
            const float2 aq = __ffma2_rn(A0, x, __ffma2_rn(A1, y, __ffma2_rn(A2, z, a0p)));
            const float2 bq = __ffma2_rn(B0, x, __ffma2_rn(B1, y, __ffma2_rn(B2, z, b0p)));
            const float2 rc = make_float2(pm_rcp_ftz(cq.x), pm_rcp_ftz(cq.y));
            const float2 ul = __fmul2_rn(aq, rc), vl = __fmul2_rn(bq, rc);
            const float2 tu = __fadd2_rd(ul, bias), tv = __fadd2_rd(vl, bias);
            const float2 fx = pm_sub2(ul, __fadd2_rn(tu, nbias)), fy = pm_sub2(vl, __fadd2_rn(tv, nbias));
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (q == 1 && !both) continue;
                // tap offset (floor(v) + V0) sw + floor(u) + U0 as below
                const unsigned xb = __float_as_uint(q ? tu.y : tu.x), yb = __float_as_uint(q ? tv.y : tv.x);
                const unsigned o = min(yb * (unsigned)sw + xb + kb, last);
                MVS_BOUND(o <= last);
                const float4 t = __ldg(qd + o);
                const float2 lo = make_float2(t.x, t.y), hi = make_float2(t.z, t.w);
                const float2 tb = __ffma2_rn(pm_dup(q ? fx.y : fx.x), pm_sub2(hi, lo), lo);   // (top, bottom)
                const float J = fmaf(q ? fy.y : fy.x, tb.y - tb.x, tb.x);
                float Jp = J - mJ, Iv = q ? iv.y : iv.x;
                if (!ALLFIN) {
                    const bool ok = Iv == Iv;
                    Jp = ok ? Jp : 0.f;
                    Iv = ok ? Iv : 0.f;
                }
                T1 += Jp;
                T2 = fmaf(Jp, Jp, T2);
                X = fmaf(Iv, Jp, X);
            }
        };
        if constexpr (Acc::FLAT) {
            constexpr int FULL = NSIDE * NSIDE / 2;
#pragma unroll PM_FLAT_AHEAD
            for (int m = 0; m < FULL; ++m) two(0, m, true);
            if (NSIDE % 2) two(0, FULL, false);
        } else {
#pragma unroll 1
            for (int row = 0; row < NSIDE; ++row)
#pragma unroll
                for (int m = 0; m < (NSIDE + 1) / 2; ++m) two(row, m, 2 * m + 1 < NSIDE);
        }
        return;
    }
    // rows rolled, the samples of a row unrolled when the side is known (the checked form, rare,
    // stays rolled to keep the instruction footprint small)
    const int side = NSIDE > 0 ? NSIDE : side_rt;
#pragma unroll 1
    for (int row = 0; row < side; ++row)
#pragma unroll((NSIDE > 0 && !CHECKED) ? NSIDE : 1)
    for (int k = 0; k < side; ++k) {
        const float4 w = win.at(row, k, row * side + k);
        const float cq = fmaf(C[0], w.x, fmaf(C[1], w.y, fmaf(C[2], w.z, c0)));
        const float aq = fmaf(A[0], w.x, fmaf(A[1], w.y, fmaf(A[2], w.z, a0)));
        const float bq = fmaf(B[0], w.x, fmaf(B[1], w.y, fmaf(B[2], w.z, b0)));
        const float rc = __fdividef(1.0f, cq);
        float ul = aq * rc, vl = bq * rc;
        bool ok = ALLFIN || w.w == w.w;
        if (CHECKED) {
            const float den = fmaf(n0, w.x, fmaf(n1, w.y, fmaf(n2, w.z, denp)));
            ok = ok && den < -1e-9f;                    // the reference skips den >= -1e-9
            ns += ok ? 1.f : 0.f;
            ok = ok && cq * __fdividef(1.0f, den) > 1e-6f && ul >= lou && ul <= hiu && vl >= lov && vl <= hiv;
            ul = ok ? ul : 0.f;
            vl = ok ? vl : 0.f;
        }
        float fu, fv;
        // top-left tap offset (floor(v) + V0) sw + floor(u) + U0 from the floor bits: one
        // multiply-add and one add of the unit's constant, wrapping exactly in 32 bits; the clamp
        // (an offset below 0 wraps above `last`) keeps every tap inside the image whatever the inputs
        const unsigned xb = pmf_floor_bits(ul, fu), yb = pmf_floor_bits(vl, fv);
        const unsigned o = min(yb * (unsigned)sw + xb + kb, last);
        MVS_BOUND(o <= last);
        const float fx = ul - fu, fy = vl - fv;
        const float4 q4 = __ldg(qd + o);
        const float t00 = q4.x, t01 = q4.z, t10 = q4.y, t11 = q4.w;
        const float top = fmaf(fx, t01 - t00, t00), bot = fmaf(fx, t11 - t10, t10);
        const float J = fmaf(fy, bot - top, top);
        if (CHECKED) ok = ok && fabsf(J) <= 3.4e38f;
        float Jp = J - mJ, Iv = w.w;
        if (CHECKED || !ALLFIN) {
            Jp = ok ? Jp : 0.f;
            Iv = ok ? Iv : 0.f;
        }
        T1 += Jp;
        T2 = fmaf(Jp, Jp, T2);
        X = fmaf(Iv, Jp, X);
        if (CHECKED) {
            S1 += Iv;
            S2 = fmaf(Iv, Iv, S2);
            cnt += ok ? 1.f : 0.f;
        }
    }
}

// float32 NCC of one (candidate, source) unit: plane (d, n) at the window's pixel, source s
// (s < S); n . ray_p = ndr < -1e-6. Follows _pm_cost: -1 below the count gate, 0 below the
// variance floor.
template <int NSIDE, class Acc>
__device__ __forceinline__ float pm_unit_ncc(const PMParams& c, const PMWinT<Acc>& wn, float rpx, float rpy, float rpz,
                                            double d, const double* n, double ndr, int sl) {
    const double num = d * ndr;
    const float n0 = (float)n[0], n1 = (float)n[1], n2 = (float)n[2], denp = (float)ndr;
    const int NW = NSIDE > 0 ? NSIDE * NSIDE : wn.nw;
    const Acc& win = wn.acc;
    const int SIDE = NSIDE > 0 ? NSIDE : wn.side;
    // ---- per (candidate, source) local map. The camera point of sample q is M ray_q / (n.ray_q),
    // M = b n^T + num R. The window centre is formed in float64 (b (n.ray_p) + num R ray_p), the
    // rows of M (which only multiply ray_q - ray_p) in float32.
    const double* p = c.par + 18 * sl;
    const double* bs = c.bsrc + 3 * sl;
    const float *pf = c.parf + 18 * sl, *bsf = c.bsf + 3 * sl;   // their float32 values
    const double rp[3] = {rpx, rpy, rpz};
    double cen[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double Rr = fma(p[3 * i], rp[0], fma(p[3 * i + 1], rp[1], p[3 * i + 2] * rp[2]));
        cen[i] = fma(bs[i], ndr, num * Rr);
    }
    const double xp = cen[0], yp = cen[1], zp = cen[2];
    const double f = p[12], pcx = p[16], pcy = p[17];
    // the centre's camera depth is zp / ndr: in front of the source needs zp < 0
    const bool front = zp < 0.0;
    const float ff = pf[12], rzf = front ? __fdividef(1.0f, (float)zp) : 0.f;
    const float ucf = fmaf(ff, (float)xp * rzf, pf[16]), vcf = fmaf(ff, (float)yp * rzf, pf[17]);
    const float Uf = fminf(fmaxf(floorf(ucf), -1048576.f), 1048576.f);
    const float Vf = fminf(fmaxf(floorf(vcf), -1048576.f), 1048576.f);
    const bool anchor = front && Uf == Uf && Vf == Vf;
    const double U0d = anchor ? (double)Uf : 0.0, V0d = anchor ? (double)Vf : 0.0;
    const double au = pcx - U0d, av = pcy - V0d;
    const float a0 = (float)fma(f, xp, au * zp), b0 = (float)fma(f, yp, av * zp), c0 = (float)zp;
    const float auf = (float)au, avf = (float)av, numf = (float)num;
    float A[3], B[3], C[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const float nj = j == 0 ? n0 : (j == 1 ? n1 : n2);
        const float mx = fmaf(bsf[0], nj, numf * pf[j]);
        const float my = fmaf(bsf[1], nj, numf * pf[3 + j]);
        const float mz = fmaf(bsf[2], nj, numf * pf[6 + j]);
        A[j] = fmaf(ff, mx, auf * mz);
        B[j] = fmaf(ff, my, avf * mz);
        C[j] = mz;
    }
    const int sw = c.iw[sl], sh = c.ih[sl];
    const float lou = (float)(-U0d), lov = (float)(-V0d);
    const float hiu = (float)(((double)sw - 1.001) - U0d), hiv = (float)(((double)sh - 1.001) - V0d);
    // integer tap position = floor bits + (U0 - magic): one add per coordinate
    const int ub = (int)U0d - 0x4B400000, vb = (int)V0d - 0x4B400000;
    const int last = sh * sw - sw - 2;                    // largest valid top-left tap offset
    // the window sums' tap offset: yb sw + xb + kb for floor bits xb, yb (unsigned, wrapping)
    const unsigned kb = (unsigned)vb * (unsigned)sw + (unsigned)ub;
    const float4* qd = c.quad[sl];
    // ---- corners: the whole window in front and inside (outside) the source (by the extremes: four
    // comparisons a unit in place of eight a corner)
    bool den_ok = true, front_all = true;
    float ul0 = 0.f, ul1 = 0.f, vl0 = 0.f, vl1 = 0.f;        // extremes over the corners, NaN if one is
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 w = win.corner(k, NW);
        const float den = fmaf(n0, w.x, fmaf(n1, w.y, fmaf(n2, w.z, denp)));
        const float cq = fmaf(C[0], w.x, fmaf(C[1], w.y, fmaf(C[2], w.z, c0)));
        const float aq = fmaf(A[0], w.x, fmaf(A[1], w.y, fmaf(A[2], w.z, a0)));
        const float bq = fmaf(B[0], w.x, fmaf(B[1], w.y, fmaf(B[2], w.z, b0)));
        const float rc = __fdividef(1.0f, cq);
        const float ul = aq * rc, vl = bq * rc;
        den_ok = den_ok && den < -1e-3f;
        front_all = front_all && cq < 1e-2f * den;
        ul0 = k ? pm_min_nan(ul0, ul) : ul;
        ul1 = k ? pm_max_nan(ul1, ul) : ul;
        vl0 = k ? pm_min_nan(vl0, vl) : vl;
        vl1 = k ? pm_max_nan(vl1, vl) : vl;
    }
    const bool known = den_ok && front_all && anchor;
    const bool inside = known && ul0 >= lou + 1.f && ul1 <= hiu - 1.f && vl0 >= lov + 1.f && vl1 <= hiv - 1.f;
    const bool outside = known && (ul1 < lou - 1.f || ul0 > hiu + 1.f || vl1 < lov - 1.f || vl0 > hiv + 1.f);
    // ---- source shift: the source at the window centre (the anchor), else 0
    float mJ = 0.f;
    if (anchor && !outside) {
        const float ul = a0 / c0, vl = b0 / c0;
        if (ul >= lou && ul <= hiu && vl >= lov && vl <= hiv) {
            float fu, fv;
            const int xi = pmf_floor(ul, fu) + ub + 0x4B400000, yi = pmf_floor(vl, fv) + vb + 0x4B400000;
            const int o = min(max(yi * sw + xi, 0), last);
            const float fx = ul - fu, fy = vl - fv;
            const float4 q4 = __ldg(qd + o);
            const float t00 = q4.x, t01 = q4.z, t10 = q4.y, t11 = q4.w;
            const float top = fmaf(fx, t01 - t00, t00), bot = fmaf(fx, t11 - t10, t10);
            const float J = fmaf(fy, bot - top, top);
            if (fabsf(J) <= 3.4e38f) mJ = J;
        }
    }
    // ---- window sums
    float T1 = 0.f, T2 = 0.f, X = 0.f, S1 = 0.f, S2 = 0.f, cnt = 0.f, ns = 0.f;
    bool checked = !den_ok;                   // the count of samples needs the per-sample test
    if (!outside && inside) {
        if (wn.allfin) {
            pm_window_sums<NSIDE, false, true>(win, SIDE, A, B, C, a0, b0, c0, n0, n1, n2, denp, lou, hiu, lov, hiv,
                                               kb, qd, sw, (unsigned)last, mJ, T1, T2, X, S1, S2, cnt, ns);
        } else {
            pm_window_sums<NSIDE, false, false>(win, SIDE, A, B, C, a0, b0, c0, n0, n1, n2, denp, lou, hiu, lov, hiv,
                                                kb, qd, sw, (unsigned)last, mJ, T1, T2, X, S1, S2, cnt, ns);
        }
        // a non-finite source value in the window poisons the sums: redo the source checked
        if (fabsf(T2) <= 3.4e38f && fabsf(X) <= 3.4e38f) {
            S1 = wn.si; S2 = wn.sii; cnt = wn.nfin;
        } else {
            checked = true;
        }
    } else if (!outside) {
        checked = true;
    }
    if (checked) {
        T1 = T2 = X = S1 = S2 = cnt = ns = 0.f;
        pm_window_sums<NSIDE, true, false>(win, SIDE, A, B, C, a0, b0, c0, n0, n1, n2, denp, lou, hiu, lov, hiv,
                                           kb, qd, sw, (unsigned)last, mJ, T1, T2, X, S1, S2, cnt, ns);
    }
    // samples counted by the reference (finite reference value, n.ray_q < -1e-9): with every
    // corner's n.ray_q < -1e-3 that is every finite sample; otherwise each lane counted them
    if (den_ok) ns = wn.nfin;
    float ncc;
    {
        if (ns < 4.f || (double)cnt < 0.7 * (double)ns) {
            ncc = -1.f;
        } else {
            const float rc = 1.0f / cnt;
            const float mi = S1 * rc, mj = T1 * rc;
            const float vi = fmaf(-mi, mi, S2 * rc), vj = fmaf(-mj, mj, T2 * rc);
            const float cv = fmaf(-mi, mj, X * rc);
            ncc = (vi < 1e-8f || vj < 1e-8f) ? 0.f : cv * rsqrtf(vi * vj);
            if (!(fabsf(ncc) <= 3.4e38f)) ncc = 0.f;
        }
    }
    return ncc;
}

// float32 photo term (top-k mean NCC) of plane (d, n): the L lanes of a pixel group evaluate one
// source each and sort their NCCs with a shuffle network; every lane returns the same value.
template <int L, int NSIDE, class Acc>
__device__ float pm_photo_lane(const PMParams& c, const PMWinT<Acc>& wn, float rpx, float rpy, float rpz, double d,
                               const double* n, double ndr, int s, unsigned gmask) {
    float ncc = s < c.S ? pm_unit_ncc<NSIDE>(c, wn, rpx, rpy, rpz, d, n, ndr, s) : -INFINITY;   // idle lanes sort last
    // ---- descending bitonic sort over the group, then the mean of the first top_k
    const int lane = threadIdx.x & (L - 1);
#pragma unroll
    for (int k = 2; k <= L; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const float o = __shfl_xor_sync(gmask, ncc, j, L);
            const bool keep_max = ((lane & k) == 0) == ((lane & j) == 0);
            ncc = keep_max ? fmaxf(ncc, o) : fminf(ncc, o);
        }
    }
    const int kk = c.top_k < c.S ? c.top_k : c.S;
    float sum = lane < kk ? ncc : 0.f;
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(gmask, sum, o, L);
    return sum / (float)kk;
}

// float32 photo term of plane (d, n) evaluated by one lane over all sources (the propagation
// step gives each lane its own candidate); the top-k list is kept sorted in registers.
template <int NSIDE, int KM, class Acc>
__device__ __forceinline__ float pm_photo_cand_k(const PMParams& c, const PMWinT<Acc>& wn, float rpx, float rpy, float rpz,
                                                 double d, const double* n, double ndr) {
    const int kk = c.top_k < c.S ? c.top_k : c.S;
    float top[KM];
#pragma unroll
    for (int q = 0; q < KM; ++q) top[q] = -INFINITY;
#pragma unroll 1
    for (int s = 0; s < c.S; ++s) {
        float x = pm_unit_ncc<NSIDE>(c, wn, rpx, rpy, rpz, d, n, ndr, s);
#pragma unroll
        for (int q = 0; q < KM; ++q) {
            if (q < kk) {
                const float hi = fmaxf(top[q], x), lo = fminf(top[q], x);
                top[q] = hi;
                x = lo;
            }
        }
    }
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < KM; ++q) sum += q < kk ? top[q] : 0.f;
    return sum / (float)kk;
}

template <int NSIDE, class Acc>
__device__ __noinline__ float pm_photo_cand_wide(const PMParams& c, const PMWinT<Acc>& wn, float rpx, float rpy, float rpz,
                                                 double d, const double* n, double ndr) {
    return pm_photo_cand_k<NSIDE, MVS_MAX_SOURCES, Acc>(c, wn, rpx, rpy, rpz, d, n, ndr);
}

// top_k <= 2 (the reference's default) keeps a 2-entry list; wider lists take an out-of-line call
template <int NSIDE, class Acc>
__device__ __forceinline__ float pm_photo_cand(const PMParams& c, const PMWinT<Acc>& wn, float rpx, float rpy, float rpz,
                                               double d, const double* n, double ndr) {
    if (c.top_k <= 2) return pm_photo_cand_k<NSIDE, 2, Acc>(c, wn, rpx, rpy, rpz, d, n, ndr);
    return pm_photo_cand_wide<NSIDE, Acc>(c, wn, rpx, rpy, rpz, d, n, ndr);
}

// Geometric term over the group: lane s contributes source s's error (float64, as pm_geo).
template <int L>
__device__ __forceinline__ double pm_geo_lane(const PMParams& c, double d, double rpx, double rpy, double rpz, int s,
                                              unsigned gmask, int ng) {
    double e = 0.0;
    if (s < c.S && c.dep[s] != nullptr) {
        const double X = c.cr0 + d * rpx, Y = c.cr1 + d * rpy, Z = c.cr2 + d * rpz;
        double u, v, z;
        e = 1.0;
        if (pm_proj(c.par + 18 * s, X, Y, Z, u, v, z)) {
            const int ui = (int)(u + 0.5), vv = (int)(v + 0.5);
            if (ui >= 0 && vv >= 0 && ui < c.iw[s] && vv < c.ih[s]) {
                const double dj = __ldg(c.dep[s] + (long long)vv * c.iw[s] + ui);
                if (isfinite(dj) && dj > 0.0) {
                    e = fabs(z - dj) / dj / c.geo_tol;
                    if (e > 1.0) e = 1.0;
                }
            }
        }
    }
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) e += __shfl_xor_sync(gmask, e, o, L);
    return e / (double)ng;
}

// Samples along one side of the window: offsets -r, -r + step, ... <= r.
__host__ __device__ inline int pm_side(int r, int step) { return (2 * r) / step + 1; }

// The lane kernel's staged window: pairs when the side is known at compile time.
template <int NSIDE>
struct PMLaneWin {
    using Acc = PMWinPairs<NSIDE>;
};
template <>
struct PMLaneWin<0> {
    using Acc = PMWinStaged;
};
// float4 entries of one pixel's staged window (nside: the compile-time side or 0; nw: its samples).
// Pairs: two entries each, the 4 corners and one more - an odd number of 16-byte units puts the
// pixels of a warp on different banks.
__host__ __device__ constexpr size_t pm_lane_entries(int nside, size_t nw) {
    return nside > 0 ? 2 * ((nside * nside + 1) / 2) + 5 : nw + 4;
}

// PHASE 0: current plane and propagation; PHASE 1: the random trials.
template <int L, int NSIDE, int PHASE>
__global__ void __launch_bounds__(256, PM_LANE_MIN_BLOCKS)
    pm_lane_kernel(const __grid_constant__ PMParams c) {
    extern __shared__ float4 pm_win[];
    const int H = c.H, W = c.W;
    const int lane = threadIdx.x & (L - 1);
    const unsigned gmask = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << (threadIdx.x & 31 & ~(L - 1));
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / L;
    int y, x;
    const bool in_img = pm_pixel(c, t, y, x);
    const long long HW = (long long)H * W, idx = (long long)y * W + x;
    if (!in_img || !c.active[idx]) {
        if (PHASE == 0 && lane == 0 && t < (long long)H * ((W + 1) / 2)) c.flags[t] = 0;
        return;
    }
    unsigned pflag = 0;
    if (PHASE == 1) {
        pflag = c.flags[t];
        if (!(pflag & 1u)) {           // no draws: the visit ends with propagation's result
            if (lane == 0) pm_finish(c, idx, c.depth[idx], c.pbest[t], c.psc[t], pflag >> 1);
            return;
        }
    }
    int ng = 0;
    for (int s = 0; s < c.S; ++s) ng += c.dep[s] != nullptr;
    const bool use_geo = c.geo_w > 0.0 && ng > 0;
    // ---- stage the window once per visit: ray offsets and reference values (NaN = no sample),
    // then the four corners of the clipped window; the window mean of the reference is the
    // shift of the float32 sums
    const int side = NSIDE > 0 ? NSIDE : pm_side(c.r, c.step);
    const int nw = side * side;
    using Acc = typename PMLaneWin<NSIDE>::Acc;
    const int entries = (int)pm_lane_entries(NSIDE, nw);
    float4* win = pm_win + (threadIdx.x / L) * entries;
    MVS_BOUND((threadIdx.x / L + 1) * entries * sizeof(float4) <= c.win_smem);
    const float rpx = __ldg(c.ray + idx), rpy = __ldg(c.ray + HW + idx), rpz = __ldg(c.ray + 2 * HW + idx);
    PMWinT<Acc> wn;
    wn.acc.w = win;
    wn.side = side;
    wn.nw = nw;
    {
        float sum = 0.f, k = 0.f;
        for (int e = lane; e < nw + 4; e += L) {
            int yy, xx;
            if (e < nw) {
                yy = y - c.r + (e / side) * c.step;
                xx = x - c.r + (e % side) * c.step;
            } else {
                const int k4 = e - nw;
                yy = k4 < 2 ? max(y - c.r, 0) : min(y + c.r, H - 1);
                xx = (k4 & 1) ? min(x + c.r, W - 1) : max(x - c.r, 0);
            }
            float4 v = make_float4(0.f, 0.f, 0.f, __int_as_float(0x7fc00000));
            if (yy >= 0 && yy < H && xx >= 0 && xx < W) {
                const long long q = (long long)yy * W + xx;
                v.x = __ldg(c.ray + q) - rpx;
                v.y = __ldg(c.ray + HW + q) - rpy;
                v.z = __ldg(c.ray + 2 * HW + q) - rpz;
                const float I = __ldg(c.ref + q);
                if (e < nw && fabsf(I) <= 3.4e38f) {
                    v.w = I;
                    sum += I;
                    k += 1.f;
                }
            }
            if constexpr (NSIDE > 0) {
                if (e < nw) {
                    float* f = reinterpret_cast<float*>(win) + Acc::slot(e);
                    f[0] = v.x;
                    f[2] = v.y;
                    f[4] = v.z;
                    f[6] = v.w;
                } else {
                    win[2 * Acc::NP + e - nw] = v;
                }
            } else {
                win[e] = v;
            }
        }
        if constexpr (NSIDE % 2 == 1 && NSIDE > 0) {   // the surplus sample of the last pair: the centre ray
            if (lane == 0) {
                float* f = reinterpret_cast<float*>(win) + Acc::slot(NSIDE * NSIDE);
                f[0] = f[2] = f[4] = f[6] = 0.f;
            }
        }
#pragma unroll
        for (int o = L >> 1; o > 0; o >>= 1) {
            sum += __shfl_xor_sync(gmask, sum, o, L);
            k += __shfl_xor_sync(gmask, k, o, L);
        }
        // shift of the float32 sums: the window mean of the reference
        const float mI = k > 0.f ? sum / k : 0.f;
        float si = 0.f, sii = 0.f;
        for (int e = lane; e < nw; e += L) {
            float* f;
            if constexpr (NSIDE > 0) f = reinterpret_cast<float*>(win) + Acc::slot(e) + 6;
            else f = &win[e].w;
            const float I = *f;
            if (I == I) {
                const float Ip = I - mI;
                *f = Ip;
                si += Ip;
                sii = fmaf(Ip, Ip, sii);
            }
        }
#pragma unroll
        for (int o = L >> 1; o > 0; o >>= 1) {
            si += __shfl_xor_sync(gmask, si, o, L);
            sii += __shfl_xor_sync(gmask, sii, o, L);
        }
        wn.nfin = k;
        wn.si = si;
        wn.sii = sii;
        wn.allfin = k == (float)nw;
        __syncwarp(gmask);
    }
    const double rx = rpx, ry = rpy, rz = rpz;
    // cost of a candidate: _pm_cost's 10 for an invalid plane, else (1 - photo) + geo_w * geo
    auto cost = [&](double d, const double* nb, double, double& photo) -> double {
        const double ndr = nb[0] * rx + nb[1] * ry + nb[2] * rz;
        if (ndr >= -1e-6 || d <= 0.0) {
            photo = 0.0;
            return 10.0;
        }
        photo = (double)pm_photo_lane<L, NSIDE>(c, wn, rpx, rpy, rpz, d, nb, ndr, lane, gmask);
        const double geo = use_geo ? pm_geo_lane<L>(c, d, rx, ry, rz, lane, gmask, ng) : 0.0;
        return (1.0 - photo) + c.geo_w * geo;
    };
    float dcur = c.depth[idx];
    float ncur[3] = {c.normal[idx], c.normal[HW + idx], c.normal[2 * HW + idx]};
    double best, sc, ph;
    unsigned long long changed = 0;
    if (PHASE == 1) {
        best = c.pbest[t];
        sc = c.psc[t];
        changed = pflag >> 1;
        pm_trials(c, c.pstate[t], dcur, ncur, best, sc, changed, cost);
        if (lane != 0) return;
        c.depth[idx] = dcur;
        c.normal[idx] = ncur[0];
        c.normal[HW + idx] = ncur[1];
        c.normal[2 * HW + idx] = ncur[2];
        pm_finish(c, idx, dcur, best, sc, changed);
        return;
    }
    const int offy[8] = {-1, 1, 0, 0, -5, 5, 0, 0};
    const int offx[8] = {0, 0, -1, 1, 0, 0, -5, 5};
    const double cached = c.cost_cache ? c.cost_cache[idx] : __longlong_as_double(0x7ff8000000000000LL);
    if (isfinite(dcur) && cached == cached) {
        best = cached;
        sc = c.score_cache[idx];
    } else if (isfinite(dcur)) {
        const double n[3] = {ncur[0], ncur[1], ncur[2]};
        best = cost((double)dcur, n, 0.0, ph);
        sc = ph;
    } else {
        best = 1e9;
        sc = -1.0;
    }
    // propagation: the neighbours' planes do not change during a colour pass, so the 8 candidate
    // costs are independent of one another. Lane k (mod L) evaluates candidate k over all sources;
    // then every lane takes the decisions in the reference's order from the shared results.
    auto cost_cand = [&](double d, const double* nb, double& photo) -> double {
        const double ndr = nb[0] * rx + nb[1] * ry + nb[2] * rz;
        if (ndr >= -1e-6 || d <= 0.0) {
            photo = 0.0;
            return 10.0;
        }
        photo = (double)pm_photo_cand<NSIDE>(c, wn, rpx, rpy, rpz, d, nb, ndr);
        const double geo = use_geo ? pm_geo(c, d, rx, ry, rz) : 0.0;
        return (1.0 - photo) + c.geo_w * geo;
    };
    constexpr int PR = (8 + L - 1) / L;          // candidates per lane
    double pcost[PR];
    float pphoto[PR], pd[PR], pn[PR][3];
    bool pok[PR];
#pragma unroll
    for (int r0 = 0; r0 < PR; ++r0) {
        const int k = r0 * L + lane;
        pok[r0] = false;
        pcost[r0] = 0.0;
        pphoto[r0] = pd[r0] = pn[r0][0] = pn[r0][1] = pn[r0][2] = 0.f;
        if (k >= 8) continue;
        const int yn = y + offy[k], xn = x + offx[k];
        if (yn < 0 || xn < 0 || yn >= H || xn >= W) continue;
        const long long nidx = (long long)yn * W + xn;
        const float dnb = c.depth[nidx];
        if (!isfinite(dnb)) continue;
        const double nb[3] = {c.normal[nidx], c.normal[HW + nidx], c.normal[2 * HW + nidx]};
        const double dn = nb[0] * __ldg(c.ray + nidx) + nb[1] * __ldg(c.ray + HW + nidx) + nb[2] * __ldg(c.ray + 2 * HW + nidx);
        const double ndr = nb[0] * rx + nb[1] * ry + nb[2] * rz;
        if (ndr >= -1e-6) continue;
        const double dp = (double)dnb * dn / ndr;
        if (dp < c.dmin || dp > c.dmax) continue;
        double phc;
        pcost[r0] = cost_cand(dp, nb, phc);
        pphoto[r0] = (float)phc;
        pd[r0] = (float)dp;
        pn[r0][0] = (float)nb[0]; pn[r0][1] = (float)nb[1]; pn[r0][2] = (float)nb[2];
        pok[r0] = true;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int from = k % L, r0 = k / L;
        const bool ok = __shfl_sync(gmask, (int)pok[r0], from, L) != 0;
        const double cst = __shfl_sync(gmask, pcost[r0], from, L);
        const float phk = __shfl_sync(gmask, pphoto[r0], from, L);
        const float dk = __shfl_sync(gmask, pd[r0], from, L);
        const float n0 = __shfl_sync(gmask, pn[r0][0], from, L);
        const float n1 = __shfl_sync(gmask, pn[r0][1], from, L);
        const float n2 = __shfl_sync(gmask, pn[r0][2], from, L);
        if (ok && cst < best) {
            best = cst;
            sc = phk;
            dcur = dk;
            ncur[0] = n0; ncur[1] = n1; ncur[2] = n2;
            ++changed;
        }
    }
    if (lane != 0) return;
    if (changed) {
        c.depth[idx] = dcur;
        c.normal[idx] = ncur[0];
        c.normal[HW + idx] = ncur[1];
        c.normal[2 * HW + idx] = ncur[2];
    }
    c.pbest[t] = best;
    c.psc[t] = sc;
    c.flags[t] = (unsigned char)((isfinite(dcur) ? 1u : 0u) | ((unsigned)changed << 1));
}

// ---------------------------------------------------------------- float32 trials, one lane per pixel
//
// In pm_lane_kernel the trials' lanes are the sources, and a pixel is seen by only some of them
// (5.1 of 8 on average in a 3 x 3 flight at 60-75 % overlap): the other lanes idle. Here a warp
// takes 32 consecutive pixels of one colour in one row and each lane evaluates its own pixel's
// two trials over all sources, as propagation evaluates its candidates; neighbouring pixels see
// the same sources, so the lanes skip the same ones together. The warp stages one tile of raw
// rays and reference values (rows y - r .. y + r, columns x_first - r .. x_last + r: 2r + 1 rows
// of 64 + 2r) in place of a window per pixel, and the window statistics are summed in the lane
// kernel's order (L strided partial sums, then its butterfly), so a trial's cost has the lane
// kernel's bits when top_k <= 2 and no source has a depth map (otherwise the top-k and geometric
// sums add the same terms in another order).
// Blocks of 4 warps; the trials of 4 iterations at 4000 x 3000, 8 sources: single samples from a tile of
// 16-byte entries (half of its wavefronts bank conflicts) 88.0 ms at 4 blocks per SM; pairs from
// planes 84.3 ms at 3 (168 registers; 82.7 with the shorter unit set-up), 89.7 ms at 4 (128, spills).
constexpr int PM_TRIAL_WARPS = 4;   // warps per block
constexpr int PM_TRIAL_MIN_BLOCKS = 3;

__host__ __device__ inline int pm_tile_pitch(int r) { return 64 + 2 * r; }
__host__ __device__ inline size_t pm_tile_entries(int r) { return (2 * (size_t)r + 1) * (64 + 2 * (size_t)r); }

// Sums over the window's samples e = 0 .. nw - 1 as an L-lane group forms them: lane l adds
// e = l, l + L, ... in order, then the xor butterfly (every lane ends with the same value).
template <int L, class F>
__device__ __forceinline__ void pm_group_sums(int nw, F&& term, float& a, float& b) {
    float pa[L], pb[L];
#pragma unroll
    for (int l = 0; l < L; ++l) {
        pa[l] = 0.f;
        pb[l] = 0.f;
        for (int e = l; e < nw; e += L) term(e, pa[l], pb[l]);
    }
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int l = 0; l < L; ++l)
            if (!(l & o)) {
                const float sa = pa[l] + pa[l | o], sb = pb[l] + pb[l | o];
                pa[l] = sa; pa[l | o] = sa;
                pb[l] = sb; pb[l | o] = sb;
            }
    a = pa[0];
    b = pb[0];
}

template <int L, int NSIDE, bool STEP1>
__global__ void __launch_bounds__(32 * PM_TRIAL_WARPS, PM_TRIAL_MIN_BLOCKS)
    pm_trial_kernel(const __grid_constant__ PMParams c) {
    extern __shared__ float4 pm_tiles[];
    const int H = c.H, W = c.W, r = c.r, step = c.step;
    const int half_w = (W + 1) / 2, wpr = (half_w + 31) >> 5;            // warps per row
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long gw = (long long)blockIdx.x * PM_TRIAL_WARPS + warp;
    if (gw >= (long long)H * wpr) return;                                 // the whole warp
    const int y = (int)(gw / wpr), k0 = (int)(gw - (long long)y * wpr) * 32;
    const int par = (y + c.colour) & 1;
    const int pitch = pm_tile_pitch(r), rows = 2 * r + 1;
    const int xs0 = 2 * k0 + par - r;                                     // image column of tile column 0
    // planes of x, y, z and reference value, each rows x pitch (pitch even: column pairs are aligned)
    const int plane = rows * pitch;
    float* tile = reinterpret_cast<float*>(pm_tiles + (size_t)warp * plane);
    MVS_BOUND((size_t)(warp + 1) * plane * sizeof(float4) <= c.win_smem);
    const long long HW = (long long)H * W;
    for (int e = lane; e < rows * pitch; e += 32) {
        const int ty = e / pitch, tx = e - ty * pitch;
        const int yy = y - r + ty, xx = xs0 + tx;
        float4 v = make_float4(0.f, 0.f, 0.f, __int_as_float(0x7fc00000));
        if (yy >= 0 && yy < H && xx >= 0 && xx < W) {
            const long long q = (long long)yy * W + xx;
            v.x = __ldg(c.ray + q);
            v.y = __ldg(c.ray + HW + q);
            v.z = __ldg(c.ray + 2 * HW + q);
            const float I = __ldg(c.ref + q);
            if (fabsf(I) <= 3.4e38f) v.w = I;
        }
        tile[e] = v.x;
        tile[plane + e] = v.y;
        tile[2 * plane + e] = v.z;
        tile[3 * plane + e] = v.w;
    }
    __syncwarp();
    const int k = k0 + lane, x = 2 * k + par;
    if (k >= half_w || x >= W) return;
    const long long t = (long long)y * half_w + k, idx = (long long)y * W + x;
    if (!c.active[idx]) return;
    const unsigned pflag = c.flags[t];
    if (!(pflag & 1u)) {               // no draws: the visit ends with propagation's result
        pm_finish(c, idx, c.depth[idx], c.pbest[t], c.psc[t], pflag >> 1);
        return;
    }
    int ng = 0;
    for (int s = 0; s < c.S; ++s) ng += c.dep[s] != nullptr;
    const bool use_geo = c.geo_w > 0.0 && ng > 0;
    const int side = NSIDE > 0 ? NSIDE : pm_side(r, step);
    const int nw = side * side;
    const float rpx = __ldg(c.ray + idx), rpy = __ldg(c.ray + HW + idx), rpz = __ldg(c.ray + 2 * HW + idx);
    // this pixel's window in the tile: sample (row, col) at w0[row * step * pitch + col * step]
    const float* w0 = tile + 2 * lane;
    const float* i0 = w0 + 3 * plane;
    const int rs = step * pitch;
    float sum, kc, si, sii;
    pm_group_sums<L>(nw, [&](int e, float& a, float& b) {
        const int row = e / side, col = e - row * side;
        const float I = i0[row * rs + col * step];
        if (I == I) {
            a += I;
            b += 1.f;
        }
    }, sum, kc);
    const float mI = kc > 0.f ? sum / kc : 0.f;
    pm_group_sums<L>(nw, [&](int e, float& a, float& b) {
        const int row = e / side, col = e - row * side;
        const float I = i0[row * rs + col * step];
        if (I == I) {
            const float Ip = I - mI;
            a += Ip;
            b = fmaf(Ip, Ip, b);
        }
    }, si, sii);
    PMWinT<PMWinTile<STEP1>> wn;
    wn.acc.t = w0;
    wn.acc.plane = plane;
    wn.acc.rs = rs;
    wn.acc.cs = step;
    wn.acc.cy0 = (max(y - r, 0) - (y - r)) * pitch;
    wn.acc.cy1 = (min(y + r, H - 1) - (y - r)) * pitch;
    wn.acc.cx0 = max(x - r, 0) - (x - r);
    wn.acc.cx1 = min(x + r, W - 1) - (x - r);
    wn.acc.rpx = rpx;
    wn.acc.rpy = rpy;
    wn.acc.rpz = rpz;
    wn.acc.mI = mI;
    wn.side = side;
    wn.nw = nw;
    wn.nfin = kc;
    wn.si = si;
    wn.sii = sii;
    wn.allfin = kc == (float)nw;
    const double rx = rpx, ry = rpy, rz = rpz;
    auto cost = [&](double d, const double* nb, double, double& photo) -> double {
        const double ndr = nb[0] * rx + nb[1] * ry + nb[2] * rz;
        if (ndr >= -1e-6 || d <= 0.0) {
            photo = 0.0;
            return 10.0;
        }
        photo = (double)pm_photo_cand<NSIDE>(c, wn, rpx, rpy, rpz, d, nb, ndr);
        const double geo = use_geo ? pm_geo(c, d, rx, ry, rz) : 0.0;
        return (1.0 - photo) + c.geo_w * geo;
    };
    float dcur = c.depth[idx];
    float ncur[3] = {c.normal[idx], c.normal[HW + idx], c.normal[2 * HW + idx]};
    double best = c.pbest[t], sc = c.psc[t];
    unsigned long long changed = pflag >> 1;
    pm_trials(c, c.pstate[t], dcur, ncur, best, sc, changed, cost);
    c.depth[idx] = dcur;
    c.normal[idx] = ncur[0];
    c.normal[HW + idx] = ncur[1];
    c.normal[2 * HW + idx] = ncur[2];
    pm_finish(c, idx, dcur, best, sc, changed);
}

}  // namespace mvs

using namespace mvs;

namespace {

// Powers of the xorshift32 step matrix: P[j] = A^(2^j), j < 64 (A^(2^j) for the stream jumps).
struct StreamTables {
    Gf2 P[64];
    PMJump J;   // J.t[j] = A^(8 * 2^j) = P[j + 3]
};

Gf2 gf2_mul(const Gf2& a, const Gf2& b) {   // (a b) e_i = a (b e_i)
    Gf2 m;
    for (int i = 0; i < 32; ++i) m.col[i] = gf2_apply(a, b.col[i]);
    return m;
}

const StreamTables& stream_tables() {
    static const StreamTables T = [] {
        StreamTables t;
        for (int i = 0; i < 32; ++i) t.P[0].col[i] = xs_step(1u << i);   // the step is linear
        for (int j = 1; j < 64; ++j) t.P[j] = gf2_mul(t.P[j - 1], t.P[j - 1]);
        for (int j = 0; j < 32; ++j) t.J.t[j] = t.P[j + 3];
        return t;
    }();
    return T;
}

}  // namespace

extern "C" uint32_t mvs_pm_stream_advance(uint32_t state, uint64_t n) {
    const StreamTables& T = stream_tables();
    for (int j = 0; n != 0; ++j, n >>= 1)
        if (n & 1u) state = gf2_apply(T.P[j], state);
    return state;
}

namespace {

size_t pm_align(size_t v) { return (v + 255) & ~(size_t)255; }

// The last of a window's offsets -r, -r + step, ... <= r.
long long pm_last(int r, int step) { return -(long long)r + 2LL * r / step * step; }

// MVS_OK and *work = false: nothing to do.
mvs_status check_pm(const mvs_pm_args* a, bool* work) {
    *work = false;
    if (!a) return fail(MVS_ERR_VALUE, "pm_refine: null arguments");
    if (a->S == 0 || a->S > MVS_MAX_SOURCES) return MVS_OK;   // the reference returns 0 here
    if (a->S < 0) return fail(MVS_ERR_VALUE, "pm_refine: negative source count");
    if (a->H < 0 || a->W < 0) return fail(MVS_ERR_VALUE, "pm_refine: negative shape");
    if (a->r < 0 || a->step < 1) return fail(MVS_ERR_VALUE, "pm_refine: needs r >= 0 and step >= 1");
    if (a->top_k < 1) return fail(MVS_ERR_VALUE, "pm_refine: top_k must be >= 1");
    if (a->H == 0 || a->W == 0 || a->iters <= 0) return MVS_OK;
    if (!a->ref || !a->ray || !a->Cr || !a->par || !a->depth || !a->normal || !a->score || !a->active)
        return fail(MVS_ERR_VALUE, "pm_refine: null pointer");
    // the step past the window's last offset is formed as an int
    if (pm_last(a->r, a->step) + a->step >= (1LL << 31))
        return fail(MVS_ERR_VALUE, "pm_refine: a window of radius %d at step %d is too large", a->r, a->step);
    if ((long long)a->H * ((a->W + 1) / 2) >= (1LL << 31))
        return fail(MVS_ERR_VALUE, "pm_refine: image of %d x %d pixels is too large", a->W, a->H);
    for (int s = 0; s < a->S; ++s) {
        if (!a->src[s]) return fail(MVS_ERR_VALUE, "pm_refine: null source %d", s);
        if (a->src_h[s] < 2 || a->src_w[s] < 2) return fail(MVS_ERR_VALUE, "pm_refine: source %d smaller than 2x2", s);
    }
    if (a->precision != MVS_PM_FP64 && a->precision != MVS_PM_FP32)
        return fail(MVS_ERR_VALUE, "pm_refine: unknown precision %d", a->precision);
    *work = true;
    return MVS_OK;
}

// Scratch of one call: per pass pixel the propagation result, its flag and stream state; per scan
// block a count; the stream state (two words, alternating passes), counts and input facts; from the
// second iteration on, the per-pixel cost cache; float64: both colours' active pixels; float32: the
// sources' footprints.
struct PMLayout {
    bool fast, use_cache;
    long long n;
    int nb;
    size_t flag_bytes, list_bytes;
    size_t o_best, o_sc, o_state, o_flags, o_bsum, o_rng, o_cache, o_list, o_quad, bytes;
};

PMLayout pm_layout(const mvs_pm_args* a) {
    PMLayout l;
    // float32 evaluation needs pinhole sources (the local map is a homography) and window positions
    // that are ints (the float64 kernel takes any)
    l.fast = a->precision == MVS_PM_FP32 && std::max(a->H, a->W) + 2LL * a->r + 64 < (1LL << 31);
    for (int s = 0; s < a->S && l.fast; ++s) {
        const double* q = a->par + 18 * s;
        l.fast = q[13] == 0.0 && q[14] == 0.0 && q[15] == 0.0;
    }
    l.use_cache = a->iters > 1;
    l.n = (long long)a->H * ((a->W + 1) / 2);
    l.nb = (int)((l.n + PM_SCAN_BLOCK - 1) / PM_SCAN_BLOCK);
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += pm_align(bytes);
        return at;
    };
    l.o_best = take(l.n * 8);
    l.o_sc = take(l.n * 8);
    l.o_state = take(l.n * 4);
    l.flag_bytes = pm_align(l.n);
    l.o_flags = take((l.fast ? 1 : 2) * l.flag_bytes);
    l.o_bsum = take((size_t)l.nb * 4);
    l.o_rng = take(256);
    l.o_cache = take(l.use_cache ? (size_t)a->H * a->W * 2 * sizeof(double) : 0);
    l.list_bytes = l.fast ? 0 : pm_align((size_t)l.n * 4);
    l.o_list = take(2 * l.list_bytes);
    l.o_quad = o;
    if (l.fast)
        for (int s = 0; s < a->S; ++s) take((size_t)a->src_w[s] * a->src_h[s] * sizeof(float4));
    l.bytes = o;
    return l;
}

}  // namespace

extern "C" size_t mvs_pm_scratch_bytes(const mvs_pm_args* a) {
    clear_error();
    bool work;
    if (check_pm(a, &work) != MVS_OK) clear_error();
    return work ? pm_layout(a).bytes : 0;
}

extern "C" mvs_status mvs_pm_refine(const mvs_pm_args* a, void* stream) {
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const size_t need = mvs_pm_scratch_bytes(a);
    void* scratch = nullptr;
    if (need) MVS_CUDA(cudaMallocAsync(&scratch, need, st), "pm_refine: scratch");
    const mvs_status s = mvs_pm_refine_ws(a, scratch, need, stream);
    if (scratch) cudaFreeAsync(scratch, st);
    return s;
}

extern "C" mvs_status mvs_pm_refine_ws(const mvs_pm_args* a, void* scratch_mem, size_t scratch_bytes, void* stream) {
    clear_error();
    bool work;
    MVS_TRY(check_pm(a, &work));
    if (!work) return MVS_OK;
    PMParams p;
    memset(&p, 0, sizeof(p));
    p.H = a->H; p.W = a->W; p.S = a->S; p.r = a->r; p.step = a->step; p.top_k = a->top_k;
    p.last = (int)pm_last(a->r, a->step);
    p.r2 = (float)a->r * (float)a->r;
    p.few = 2LL * a->r / a->step + 1 <= 20;
    p.cr0 = a->Cr[0]; p.cr1 = a->Cr[1]; p.cr2 = a->Cr[2];
    p.geo_w = a->geo_w; p.geo_tol = a->geo_tol; p.dmin = a->dmin; p.dmax = a->dmax;
    p.ref = a->ref; p.ray = a->ray; p.depth = a->depth; p.normal = a->normal; p.score = a->score;
    p.active = a->active;
    p.changed = reinterpret_cast<unsigned long long*>(a->changed);
    for (int s = 0; s < a->S; ++s) {
        p.img[s] = a->src[s];
        p.dep[s] = a->src_depth[s];
        p.iw[s] = a->src_w[s];
        p.ih[s] = a->src_h[s];
        for (int k = 0; k < 18; ++k) p.par[18 * s + k] = a->par[18 * s + k];
        p.pinhole[s] = a->par[18 * s + 13] == 0.0 && a->par[18 * s + 14] == 0.0 && a->par[18 * s + 15] == 0.0;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const long long HW = (long long)a->H * a->W;
    const PMLayout lay = pm_layout(a);
    const bool fast = lay.fast;
    {
        for (int s = 0; s < a->S; ++s) {
            const double* q = a->par + 18 * s;
            // b_s = R_s (C_ref - C_s)
            const double e0 = a->Cr[0] - q[9], e1 = a->Cr[1] - q[10], e2 = a->Cr[2] - q[11];
            for (int i = 0; i < 3; ++i) {
                p.bsrc[3 * s + i] = q[3 * i] * e0 + q[3 * i + 1] * e1 + q[3 * i + 2] * e2;
                p.bsf[3 * s + i] = (float)p.bsrc[3 * s + i];
            }
            for (int k = 0; k < 18; ++k) p.parf[18 * s + k] = (float)q[k];
        }
    }
    if (!scratch_mem || scratch_bytes < lay.bytes)
        return fail(MVS_ERR_VALUE, "pm_refine: scratch of %zu bytes below the %zu needed", scratch_bytes, lay.bytes);
    char* scratch = reinterpret_cast<char*>(scratch_mem);
    const long long n = lay.n;
    const int nb = lay.nb;
    const bool use_cache = lay.use_cache;
    p.pbest = reinterpret_cast<double*>(scratch + lay.o_best);
    p.psc = reinterpret_cast<double*>(scratch + lay.o_sc);
    unsigned* pstate = reinterpret_cast<unsigned*>(scratch + lay.o_state);
    p.pstate = pstate;
    p.flags = reinterpret_cast<unsigned char*>(scratch + lay.o_flags);
    unsigned* bsum = reinterpret_cast<unsigned*>(scratch + lay.o_bsum);
    unsigned* rng = reinterpret_cast<unsigned*>(scratch + lay.o_rng);
    if (use_cache) {
        p.cost_cache = reinterpret_cast<double*>(scratch + lay.o_cache);
        p.score_cache = p.cost_cache + HW;
        cudaMemsetAsync(p.cost_cache, 0xFF, (size_t)HW * sizeof(double), st);   // all-ones = NaN: recompute
    }
    if (fast) {
        size_t off = lay.o_quad;
        for (int s = 0; s < a->S; ++s) {
            float4* q = reinterpret_cast<float4*>(scratch + off);
            p.quad[s] = q;
            off += pm_align((size_t)a->src_w[s] * a->src_h[s] * sizeof(float4));
            const long long ns = (long long)a->src_w[s] * a->src_h[s];
            const int qb = (int)std::min<long long>((ns + 255) / 256, num_sms() * 8LL);
            pm_quad_kernel<<<qb, 256, 0, st>>>(a->src[s], a->src_w[s], a->src_h[s], q);
        }
    }
    unsigned char* flags = reinterpret_cast<unsigned char*>(scratch + lay.o_flags);
    if (!fast) {
        // pixels that are not active never draw; the input facts and both colours' active pixels
        cudaMemsetAsync(flags, 0, 2 * lay.flag_bytes, st);
        PMStats* stats = reinterpret_cast<PMStats*>(rng + 8);
        cudaMemsetAsync(stats, 0, sizeof(PMStats), st);
        p.stats = stats;
        const unsigned sb = num_sms() * 8;
        pm_bend_kernel<<<sb, 256, 0, st>>>(a->ray, a->H, a->W, stats);
        pm_stats_kernel<<<sb, 256, 0, st>>>(a->ref, HW, stats);
        for (int s = 0; s < a->S; ++s)
            pm_stats_kernel<<<sb, 256, 0, st>>>(a->src[s], (long long)a->src_w[s] * a->src_h[s], stats);
        for (int colour = 0; colour < 2; ++colour) {
            unsigned* list = reinterpret_cast<unsigned*>(scratch + lay.o_list + colour * lay.list_bytes);
            pm_active_count_kernel<<<nb, PM_SCAN_BLOCK, 0, st>>>(a->active, a->H, a->W, colour, bsum);
            pm_offsets_kernel<<<1, PM_SCAN_BLOCK, 0, st>>>(bsum, nb, rng + 4 + colour);
            pm_active_list_kernel<<<nb, PM_SCAN_BLOCK, 0, st>>>(a->active, a->H, a->W, colour, bsum, list);
        }
    }
    const PMJump& J = stream_tables().J;
    // float32 lanes: one per source; a block holds as many pixel groups as its staged windows fit
    const int lanes = a->S <= 4 ? 4 : (a->S <= 8 ? 8 : 16);
    const int side = fast ? pm_side(a->r, a->step) : 0;
    const size_t win_bytes = pm_lane_entries(side == 7 || side == 5 ? side : 0, (size_t)side * side) * sizeof(float4);
    int groups = 256 / lanes;
    while (groups > 1 && (size_t)groups * win_bytes > 96 * 1024) groups >>= 1;
    const int block = fast ? groups * lanes : 128;
    const size_t smem = fast ? (size_t)groups * win_bytes : 0;
    p.win_smem = (unsigned)smem;
    void (*lane_kernel[2])(PMParams) = {nullptr, nullptr};
    mvs_status status = MVS_OK;
    if (fast) {
#define PM_PICK(LN, PH)                                                                           \
    lane_kernel[PH] = side == 7 ? pm_lane_kernel<LN, 7, PH> : side == 5 ? pm_lane_kernel<LN, 5, PH> \
                                                            : pm_lane_kernel<LN, 0, PH>;
        if (lanes == 4) { PM_PICK(4, 0) PM_PICK(4, 1) }
        else if (lanes == 8) { PM_PICK(8, 0) PM_PICK(8, 1) }
        else { PM_PICK(16, 0) PM_PICK(16, 1) }
#undef PM_PICK
        for (int ph = 0; ph < 2 && status == MVS_OK; ++ph)
            status = allow_smem(lane_kernel[ph], smem, "pm_refine: shared-memory carve-out");
    }
    // the trials: one lane per pixel (pm_trial_kernel) when the warps' tiles fit in shared memory,
    // else the lane groups' kernel
    void (*trial_kernel)(PMParams) = nullptr;
    const size_t smem_trial = (size_t)PM_TRIAL_WARPS * pm_tile_entries(a->r) * sizeof(float4);
    const int wpr = (int)(((a->W + 1) / 2 + 31) / 32);
    const unsigned grid_trial = (unsigned)(((long long)a->H * wpr + PM_TRIAL_WARPS - 1) / PM_TRIAL_WARPS);
    if (fast && status == MVS_OK && smem_trial <= MVS_SMEM_MAX) {
#define PM_PICK_TRIAL(LN)                                                                        \
    trial_kernel = side == 7 && a->step == 1   ? pm_trial_kernel<LN, 7, true>                       \
                   : side == 5 && a->step == 1 ? pm_trial_kernel<LN, 5, true>                       \
                   : side == 7                 ? pm_trial_kernel<LN, 7, false>                      \
                   : side == 5                 ? pm_trial_kernel<LN, 5, false>                      \
                                               : pm_trial_kernel<LN, 0, false>;
        if (lanes == 4) { PM_PICK_TRIAL(4) }
        else if (lanes == 8) { PM_PICK_TRIAL(8) }
        else { PM_PICK_TRIAL(16) }
#undef PM_PICK_TRIAL
        if (allow_smem(trial_kernel, smem_trial, "pm_refine: trials") != MVS_OK) {
            cudaGetLastError();
            clear_error();
            trial_kernel = nullptr;
        }
    }
    const unsigned grid = fast ? (unsigned)((n * lanes + block - 1) / block) : (unsigned)((n + 127) / 128);
    if (status == MVS_OK) {
        pm_rng_init_kernel<<<1, 1, 0, st>>>(rng, a->rng_state, a->seed | 1u);
        status = check_launch("pm_refine: stream start");
    }
    int cur = 0;
    for (int it = 0; it < a->iters && status == MVS_OK; ++it) {
        const int git = a->it0 + it;
        p.it = git;
        p.dd_scale = 0.05 / (double)(git + 1);
        p.nn_scale = 0.3 / (double)(git + 1);
        for (int colour = 0; colour < 2 && status == MVS_OK; ++colour) {
            p.colour = colour;
            if (!fast) {
                p.flags = flags + colour * lay.flag_bytes;
                p.list = reinterpret_cast<unsigned*>(scratch + lay.o_list + colour * lay.list_bytes);
                p.n_list = rng + 4 + colour;
            }
            p.win_smem = (unsigned)smem;
            if (fast) lane_kernel[0]<<<grid, block, smem, st>>>(p);
            else {
                pm_kernel<PM_CURRENT><<<grid, 128, 0, st>>>(p);
                pm_kernel<PM_PROPAGATE><<<(unsigned)((n * 8 + 127) / 128), 128, 0, st>>>(p);
            }
            pm_count_kernel<<<nb, PM_SCAN_BLOCK, 0, st>>>(p.flags, n, bsum);
            pm_scan_kernel<<<1, PM_SCAN_BLOCK, 0, st>>>(bsum, nb, rng, cur, cur ^ 1, J);
            pm_state_kernel<<<nb, PM_SCAN_BLOCK, 0, st>>>(p.flags, n, bsum, rng, cur, J, pstate);
            if (trial_kernel) {
                p.win_smem = (unsigned)smem_trial;
                trial_kernel<<<grid_trial, 32 * PM_TRIAL_WARPS, smem_trial, st>>>(p);
            } else if (fast) {
                lane_kernel[1]<<<grid, block, smem, st>>>(p);
            }
            else pm_kernel<PM_TRIALS><<<grid, 128, 0, st>>>(p);
            cur ^= 1;
            status = check_launch("pm_refine kernels");
        }
    }
    if (status == MVS_OK && a->rng_state) {
        if (cudaMemcpyAsync(a->rng_state, rng + cur, sizeof(unsigned), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            status = fail(MVS_ERR_CUDA, "pm_refine: stream state copy");
    }
    return status;
}

namespace mvs {
__global__ void quotients_kernel(long long n, const double* a, const double* b, double* quot, double* rcp) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const double r = rcp_newton(b[i]);
    rcp[i] = r;
    quot[i] = pm_quot(a[i], b[i], r);
}
}  // namespace mvs

extern "C" mvs_status mvs_debug_quotients(int64_t n, const double* a, const double* b, double* quot, double* rcp,
                                          void* stream) {
    clear_error();
    if (n < 0) return fail(MVS_ERR_VALUE, "quotients: negative size");
    if (n == 0) return MVS_OK;
    if (!a || !b || !quot || !rcp) return fail(MVS_ERR_VALUE, "quotients: null pointer");
    quotients_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(n, a, b, quot, rcp);
    return check_launch("quotients");
}

unsigned mvs::take_bound_violations_pm() { return take_bound_violations_here(); }
