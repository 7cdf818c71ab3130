// The legacy ground-grid height sweep of the reference (mvs.dense_reconstruct, mvs.py:138-434) on
// the device: the view sampler (_mvs.sample_view, _mvs.pyx:13-58, the CPU twin of the CuPy kernel
// in _cuda.py:88-124), the float64 summed-area box mean (_fast.box_sat_mean, _fast.pyx:897-942),
// the photo-consistency score of a stack of height hypotheses (score_at, mvs.py:254-304) and the
// 8-path semi-global aggregation (_mvs.sgm, _mvs.pyx:98-251).
//
// This file is compiled with -fmad=false: every float64 / float32 expression is evaluated with one
// rounding per operation in the written order, as the reference's C and NumPy evaluate it, so the
// sampler, the box means and the aggregation are bit-identical to the reference's.
#include "common.cuh"

namespace mvs {

// ---------------------------------------------------------------- sampler
struct SampleParams {
    int h, w, nch, D, H, W;
    double R[9], C[3], f, k1, k2, k3, cx, cy, X0, Y0, gsd;
    const float* img;
    const float* Z;
    float* out;
    unsigned char* valid;
};

__global__ void __launch_bounds__(256) sample_view_kernel(const __grid_constant__ SampleParams p) {
    const long long n = (long long)p.D * p.H * p.W;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = (int)(i % p.W);
    const int r = (int)((i / p.W) % p.H);
    const double Y = p.Y0 - ((double)r + 0.5) * p.gsd;
    const double X = p.X0 + ((double)c + 0.5) * p.gsd;
    const double dx = X - p.C[0], dy = Y - p.C[1], dz = (double)p.Z[i] - p.C[2];
    const double zc = p.R[6] * dx + p.R[7] * dy + p.R[8] * dz;
    float* o = p.out + i * p.nch;
    bool ok = zc > 1e-6;
    double u = 0.0, v = 0.0;
    if (ok) {
        const double xc = p.R[0] * dx + p.R[1] * dy + p.R[2] * dz;
        const double yc = p.R[3] * dx + p.R[4] * dy + p.R[5] * dz;
        const double nx = xc / zc, ny = yc / zc;
        const double r2 = nx * nx + ny * ny;
        const double d = 1.0 + r2 * (p.k1 + r2 * (p.k2 + r2 * p.k3));
        u = p.f * d * nx + p.cx;
        v = p.f * d * ny + p.cy;
        // NaN positions fail every comparison of the reference's test and are sampled there as
        // garbage; here they are invalid
        ok = u >= 0.0 && v >= 0.0 && u <= (double)(p.w - 1) && v <= (double)(p.h - 1);
    }
    if (!ok) {
        for (int ch = 0; ch < p.nch; ++ch) o[ch] = 0.f;
        p.valid[i] = 0;
        return;
    }
    const int x0 = (int)u, y0 = (int)v;
    const int x1 = x0 + 1 < p.w ? x0 + 1 : x0, y1 = y0 + 1 < p.h ? y0 + 1 : y0;
    const double fx = u - (double)x0, fy = v - (double)y0;
    for (int ch = 0; ch < p.nch; ++ch) {
        const double a00 = p.img[((long long)y0 * p.w + x0) * p.nch + ch];
        const double a01 = p.img[((long long)y0 * p.w + x1) * p.nch + ch];
        const double a10 = p.img[((long long)y1 * p.w + x0) * p.nch + ch];
        const double a11 = p.img[((long long)y1 * p.w + x1) * p.nch + ch];
        o[ch] = (float)((1 - fy) * ((1 - fx) * a00 + fx * a01) + fy * ((1 - fx) * a10 + fx * a11));
    }
    p.valid[i] = 1;
}

// ---------------------------------------------------------------- float64 summed-area box mean
// Padded table S (PH = H + 2r + 1 rows, PW = W + 2r + 1 columns) per plane, built as the reference
// builds its ring rows: column sums down the rows (one thread per column), then a running total of
// those along each row (one thread per row); the window mean takes the four corners in the
// reference's order.
__global__ void box_cols_kernel(int B, int H, int W, int r, const float* __restrict__ a, double* __restrict__ cs) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)B * W) return;
    const int b = (int)(t / W), x = (int)(t - (long long)b * W);
    const int PH = H + 2 * r + 1;
    const float* ab = a + (long long)b * H * W;
    double* cb = cs + (long long)b * PH * W;
    double col = 0.0;
    for (int i = 0; i < PH; ++i) {
        const int ay = i - r - 1;
        const double val = (ay >= 0 && ay < H) ? (double)ab[(long long)ay * W + x] : 0.0;
        col = col + val;
        cb[(long long)i * W + x] = col;
    }
}

__global__ void box_rows_kernel(int B, int H, int W, int r, const double* __restrict__ cs, double* __restrict__ sat) {
    const int PH = H + 2 * r + 1, PW = W + 2 * r + 1;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)B * PH) return;
    const long long b = t / PH, i = t - b * PH;
    const double* row = cs + (b * PH + i) * W;
    double* cur = sat + (b * PH + i) * PW;
    double total = 0.0;
    for (int x = 0; x < r + 1; ++x) cur[x] = 0.0;
    for (int x = 0; x < W; ++x) {
        total = total + row[x];
        cur[x + r + 1] = total;
    }
    for (int x = r + 1 + W; x < PW; ++x) cur[x] = total;
}

__global__ void box_mean_kernel(int B, int H, int W, int r, const double* __restrict__ sat, float* __restrict__ out) {
    const long long n = (long long)B * H * W;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int k = 2 * r + 1, PH = H + 2 * r + 1, PW = W + 2 * r + 1;
    const int x = (int)(t % W);
    const int y = (int)((t / W) % H);
    const long long b = t / ((long long)H * W);
    const double* cur = sat + (b * PH + y + k) * PW;
    const double* old = sat + (b * PH + y) * PW;
    double val = cur[x + k] - old[x + k];
    val = val - cur[x];
    val = val + old[x];
    out[t] = (float)(val / ((double)k * (double)k));
}

// ---------------------------------------------------------------- score of height hypotheses
// score_at (mvs.py:254-304) after the sampling and the box means, for every cell of a (D, H, W)
// hypothesis stack and V views: the cell's reference view is the nearest camera (in X, Y) among
// those whose window is fully valid; the NCC of every other view against it (box statistics,
// variance floor 1e-6, -1 where either window is not full), the mean of the topk largest, scaled
// by the reference's texture strength. Arrays are (V or pairs, D, H, W) float32 planes:
//   M (box of S), S2 (box of S*S), VA (box of the valid mask), PP (box of S_a * S_b for the pairs
//   a < b in np.triu_indices order).
struct ScoreParams {
    int V, D, H, W, topk;
    float full, min_texture, full_texture;
    const float* M;
    const float* S2;
    const float* VA;
    const float* PP;
    const float* cxs;                 // (W) float32 cell centres, X
    const float* cys;                 // (H) float32 cell centres, Y
    float camx[16], camy[16];         // the views' centres, rounded to float32
    float* score;                     // (D, H, W)
    float* st;                        // (V, D, H, W) NCC against the cell's reference (-2: itself), or null
    int* ref;                         // (D, H, W) reference view, or null
};

__device__ __forceinline__ int pair_slot(int a, int b, int V) {   // np.triu_indices(V, 1) order, a < b
    return a * V - a * (a + 1) / 2 + (b - a - 1);
}

__global__ void __launch_bounds__(256) height_score_kernel(const __grid_constant__ ScoreParams p) {
    const long long plane = (long long)p.D * p.H * p.W;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= plane) return;
    const int x = (int)(i % p.W);
    const int y = (int)((i / p.W) % p.H);
    const int V = p.V;
    float var[16];
    bool full[16];
    // reference: argmin over views of (full ? d2 : inf), first index on ties (np.argmin)
    int ref = 0;
    float dmin = INFINITY;
    for (int v = 0; v < V; ++v) {
        const float m = p.M[v * plane + i];
        var[v] = __fsub_rn(p.S2[v * plane + i], __fmul_rn(m, m));
        full[v] = p.VA[v * plane + i] >= p.full;
        const float ey = __fsub_rn(p.cys[y], p.camy[v]), ex = __fsub_rn(p.cxs[x], p.camx[v]);
        const float d2 = __fadd_rn(__fmul_rn(ey, ey), __fmul_rn(ex, ex));
        const float dist = full[v] ? d2 : INFINITY;
        if (v == 0 || dist < dmin) {
            dmin = dist;
            ref = v;
        }
    }
    // NCC(ref, v) for every view
    float st[16];
    for (int v = 0; v < V; ++v) {
        if (v == ref) {
            st[v] = -2.f;
            continue;
        }
        const int a = min(ref, v), b = max(ref, v);
        const float cov = __fsub_rn(p.PP[pair_slot(a, b, V) * plane + i], __fmul_rn(p.M[a * plane + i], p.M[b * plane + i]));
        const float va = fmaxf(var[a], 1e-6f), vb = fmaxf(var[b], 1e-6f);
        const float ncc = __fdiv_rn(cov, __fsqrt_rn(__fmul_rn(va, vb)));
        st[v] = (full[a] && full[b]) ? ncc : -1.f;
    }
    if (p.st)
        for (int v = 0; v < V; ++v) p.st[v * plane + i] = st[v];
    // mean of the topk largest (summed in descending order)
    float top[16];
    for (int v = 0; v < V; ++v) top[v] = st[v];
    for (int a = 1; a < V; ++a) {                        // insertion sort, descending
        const float t = top[a];
        int b = a - 1;
        while (b >= 0 && top[b] < t) {
            top[b + 1] = top[b];
            --b;
        }
        top[b + 1] = t;
    }
    float sum = 0.f;
    for (int k = 0; k < p.topk; ++k) sum = __fadd_rn(sum, top[k]);
    float score = __fdiv_rn(sum, (float)p.topk);
    const float varR = var[ref];
    float tex = __fdiv_rn(__fsqrt_rn(fmaxf(varR, 0.f)), p.full_texture);
    tex = fminf(fmaxf(tex, 0.f), 1.f);
    const bool ok = isfinite(dmin) && varR > p.min_texture;
    p.score[i] = ok ? __fmul_rn(score, tex) : 0.f;
    if (p.ref) p.ref[i] = ref;
}

// ---------------------------------------------------------------- one score evaluation in three launches
// mvs_height_eval: every view's samples, all window means, the score. The views' samples come from one
// launch; the window means read the samples (and form squares and pair products as they read, in
// float32 as the separate arrays would hold them) instead of 2 V + V (V - 1) / 2 written copies.

struct EvalView {
    const float* img;                 // (h, w) grey
    int h, w;
    double R[9], C[3], f, k1, k2, k3, cx, cy;
};
struct EvalParams {
    int V, D, H, W;
    double X0, Y0, gsd;
    const float* Z;                   // (D, H, W)
    float* S;                         // (V, D, H, W)
    unsigned char* valid;             // (V, D, H, W)
    EvalView view[16];
};

// blockIdx.y: the view. The arithmetic is sample_view_kernel's.
__global__ void __launch_bounds__(256) height_sample_kernel(const __grid_constant__ EvalParams p) {
    const long long n = (long long)p.D * p.H * p.W;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const EvalView& c = p.view[blockIdx.y];
    const int x = (int)(i % p.W), y = (int)((i / p.W) % p.H);
    const double Y = p.Y0 - ((double)y + 0.5) * p.gsd;
    const double X = p.X0 + ((double)x + 0.5) * p.gsd;
    const double dx = X - c.C[0], dy = Y - c.C[1], dz = (double)p.Z[i] - c.C[2];
    const double zc = c.R[6] * dx + c.R[7] * dy + c.R[8] * dz;
    const long long o = blockIdx.y * n + i;
    bool ok = zc > 1e-6;
    double u = 0.0, v = 0.0;
    if (ok) {
        const double xc = c.R[0] * dx + c.R[1] * dy + c.R[2] * dz;
        const double yc = c.R[3] * dx + c.R[4] * dy + c.R[5] * dz;
        const double nx = xc / zc, ny = yc / zc;
        const double r2 = nx * nx + ny * ny;
        const double d = 1.0 + r2 * (c.k1 + r2 * (c.k2 + r2 * c.k3));
        u = c.f * d * nx + c.cx;
        v = c.f * d * ny + c.cy;
        ok = u >= 0.0 && v >= 0.0 && u <= (double)(c.w - 1) && v <= (double)(c.h - 1);
    }
    p.valid[o] = ok ? 1 : 0;
    if (!ok) {
        p.S[o] = 0.f;
        return;
    }
    const int x0 = (int)u, y0 = (int)v;
    const int x1 = x0 + 1 < c.w ? x0 + 1 : x0, y1 = y0 + 1 < c.h ? y0 + 1 : y0;
    const double fx = u - (double)x0, fy = v - (double)y0;
    const float *r0 = c.img + (long long)y0 * c.w, *r1 = c.img + (long long)y1 * c.w;
    const double a00 = __ldg(r0 + x0), a01 = __ldg(r0 + x1), a10 = __ldg(r1 + x0), a11 = __ldg(r1 + x1);
    p.S[o] = (float)((1 - fy) * ((1 - fx) * a00 + fx * a01) + fy * ((1 - fx) * a10 + fx * a11));
}

// The plane of the score's window means: 0 .. V-1 samples, V .. 2V-1 their squares, 2V .. 3V-1 the valid
// masks, then the pair products in np.triu_indices order.
struct EvalPlane {
    const float* a;
    const float* b;                   // product a * b, or null
    const unsigned char* m;           // mask instead
    __device__ __forceinline__ double at(long long i) const {
        if (m) return (double)(float)m[i];
        const float v = __ldg(a + i);
        return (double)(b ? v * __ldg(b + i) : v);
    }
};

// Window means by the reference's float64 summed-area table (see box_cols_kernel): one block per plane
// moves down its rows by 32. Threads are columns for the column sums, a warp's lanes are rows for the
// row totals, and a ring of 32 + k table rows in shared memory feeds the four corners, so the table
// (16 bytes a cell, written and read twice) never leaves the SM. Every sum runs in the order of the
// separate passes. Needs the ring in shared memory (height_box_smem); wider grids take the passes.
// Bound by the serial float64 sums and, before, by integer divisions around them: over a 9-view flight's
// 80 evaluations 4.9 ms (7.4 ms with a slot by modulo, a cell by division and the mean by a float64
// division), where the three passes took 7.4 ms and ~4 ms for the stacked, squared, gathered and
// multiplied copies that fed them.
constexpr int HB_ROWS = 32, HB_AHEAD = 8;      // rows per step; rows whose loads are in flight together
static size_t height_box_smem(int W, int r) {      // (the factors as 64 bits: 2 r may pass 2^31)
    return ((size_t)HB_ROWS + 2 * (size_t)r + 1) * ((size_t)W + 1) * sizeof(double);
}

__global__ void __launch_bounds__(256) height_box_kernel(const __grid_constant__ EvalParams p, int r,
                                                         float* __restrict__ out) {
    extern __shared__ double hb_ring[];
    const int V = p.V, H = p.H, W = p.W, k = 2 * r + 1, RING = HB_ROWS + k, pitch = W + 1;
    const int q = blockIdx.x, d = blockIdx.y;
    const long long HW = (long long)H * W, DHW = (long long)p.D * HW;
    EvalPlane pl;
    pl.b = nullptr;
    pl.m = nullptr;
    if (q < 2 * V) {
        const int v = q % V;
        pl.a = p.S + v * DHW + d * HW;
        if (q >= V) pl.b = pl.a;
    } else if (q < 3 * V) {
        pl.a = nullptr;
        pl.m = p.valid + (q - 2 * V) * DHW + d * HW;
    } else {
        int e = q - 3 * V, a = 0;
        while (e >= V - 1 - a) {
            e -= V - 1 - a;
            ++a;
        }
        pl.a = p.S + a * DHW + d * HW;
        pl.b = p.S + (a + 1 + e) * DHW + d * HW;
    }
    float* o = out + ((long long)q * p.D + d) * HW;
    const double kk = (double)k * (double)k, rk = 1.0 / kk;
    // table row i (0 .. H + 2 r, padded; the first r + 1 are zeros) lives in ring slot i mod RING; column
    // sums of each thread's columns stay in registers from row to row
    constexpr int MAXC = 4;                       // columns per thread (W <= 4 * 256)
    double col[MAXC];
#pragma unroll
    for (int m = 0; m < MAXC; ++m) col[m] = 0.0;
    const int PH = H + k;
    int base = 0;                                 // slot of row i0
    auto slot = [&](int ahead) {                  // of row i0 + ahead, -RING <= ahead < RING
        const int q = base + ahead;
        return q >= RING ? q - RING : (q < 0 ? q + RING : q);
    };
    for (int i0 = 0; i0 < PH; i0 += HB_ROWS) {
        const int rows = min(HB_ROWS, PH - i0);
        // column sums of rows i0 .. i0 + rows - 1 (padded row i is image row i - r - 1)
#pragma unroll
        for (int m = 0; m < MAXC; ++m) {
            const int x = threadIdx.x + m * 256;
            if (x < W) {
                double c = col[m];
                for (int a = 0; a < rows; a += HB_AHEAD) {
                    // (rows past the image are read at its edge and count as 0)
                    double v[HB_AHEAD];
#pragma unroll
                    for (int u = 0; u < HB_AHEAD; ++u)
                        v[u] = pl.at((long long)min(max(i0 + a + u - r - 1, 0), H - 1) * W + x);
#pragma unroll
                    for (int u = 0; u < HB_AHEAD; ++u) {
                        const int ay = i0 + a + u - r - 1;
                        if (a + u < rows) {
                            c = c + ((ay >= 0 && ay < H) ? v[u] : 0.0);
                            hb_ring[slot(a + u) * pitch + x] = c;
                        }
                    }
                }
                col[m] = c;
            }
        }
        __syncthreads();
        // running totals along the rows, in place: lane = row
        if ((int)threadIdx.x < rows) {
            double* row = hb_ring + slot(threadIdx.x) * pitch;
            double total = 0.0;
            int x = 0;
            for (; x + 8 <= W; x += 8) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = row[x + u];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    total = total + v[u];
                    row[x + u] = total;
                }
            }
            for (; x < W; ++x) {
                total = total + row[x];
                row[x] = total;
            }
        }
        __syncthreads();
        // the means whose lower table row is one of these, y = i - k: 4 rows of 64 threads at a time
        for (int a = threadIdx.x >> 6; a < rows; a += 4) {
            const int y = i0 + a - k;
            if (y < 0) continue;
            const double* cur = hb_ring + slot(a) * pitch;
            const double* old = hb_ring + slot(a - k) * pitch;
            for (int x = threadIdx.x & 63; x < W; x += 64) {
                // padded column j holds the total up to image column j - r - 1 (0 before it, the last after)
                const int jl = x - r - 1, jr = min(x + r, W - 1);
                double val = cur[jr] - old[jr];
                val = val - (jl >= 0 ? cur[jl] : 0.0);
                val = val + (jl >= 0 ? old[jl] : 0.0);
                // val / kk: the quotient's remainder is exact in one fused operation (Markstein)
                const double t = val * rk;
                o[(long long)y * W + x] = (float)(isfinite(t) ? __fma_rn(__fma_rn(-t, kk, val), rk, t) : t);
            }
        }
        __syncthreads();
        base = slot(HB_ROWS);                     // (HB_ROWS < RING)
    }
}

// ---------------------------------------------------------------- refinement of a coarser surface
// The refinement's steps around the score, each in NumPy's / torch's float32 order: the upsampled
// surface and its height stack, the choice among the scores with the parabola, the 3 x 3 median.

// up = the coarser surface (hc, wc) repeated 2 x 2, cropped to (H, W) or padded with its edge; stack[k] =
// up + offs[k].
__global__ void __launch_bounds__(256) height_stack_kernel(int H, int W, int hc, int wc, int K, const float* __restrict__ Zc,
                                                           const float* __restrict__ offs, float* __restrict__ up,
                                                           float* __restrict__ stack) {
    const long long HW = (long long)H * W, i = blockIdx.x * 256LL + threadIdx.x;
    if (i >= HW) return;
    const int y = (int)i / W, x = (int)i - y * W;            // (H W < 2^31)
    const float z = Zc[(long long)min(y >> 1, hc - 1) * wc + min(x >> 1, wc - 1)];
    up[i] = z;
    for (int k = 0; k < K; ++k) stack[k * HW + i] = __fadd_rn(z, __ldg(offs + k));
}

// The first best score's hypothesis; a best score below `weak` keeps the middle one; `parabola`: the
// vertex through its neighbours' scores. out = (up + offs[b]) + frac * cell.
__global__ void __launch_bounds__(256) height_pick_kernel(long long HW, int K, const float* __restrict__ sc,
                                                          const float* __restrict__ up, const float* __restrict__ offs,
                                                          float weak, int parabola, float cell, float* __restrict__ out) {
    const long long i = blockIdx.x * 256LL + threadIdx.x;
    if (i >= HW) return;
    int b = 0;
    float best = sc[i];
    for (int k = 1; k < K; ++k) {
        const float v = sc[k * HW + i];
        if (v > best || (v != v && best == best)) {      // a NaN counts as the largest, the first one wins
            best = v;
            b = k;
        }
    }
    if (best < weak) {
        b = K / 2;
        best = sc[b * HW + i];
    }
    float frac = 0.f;
    if (parabola) {
        const float lo = sc[max(b - 1, 0) * HW + i], hi = sc[min(b + 1, K - 1) * HW + i];
        const float den = __fadd_rn(__fsub_rn(lo, __fmul_rn(2.f, best)), hi);
        if (den < -1e-6f && b > 0 && b < K - 1) {
            const float f = __fdiv_rn(__fmul_rn(0.5f, __fsub_rn(lo, hi)), den);
            frac = f < -0.5f ? -0.5f : (f > 0.5f ? 0.5f : f);
        }
    }
    out[i] = __fadd_rn(__fadd_rn(up[i], __ldg(offs + b)), __fmul_rn(frac, cell));
}

// 3 x 3 median with edge padding; NaN sorts last.
__global__ void __launch_bounds__(256) median3_kernel(int H, int W, const float* __restrict__ a, float* __restrict__ out) {
    const long long i = blockIdx.x * 256LL + threadIdx.x;
    if (i >= (long long)H * W) return;
    const int y = (int)i / W, x = (int)i - y * W;            // (H W < 2^31)
    float v[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
        v[k] = a[(long long)min(max(y + (k / 3 - 1), 0), H - 1) * W + min(max(x + (k % 3 - 1), 0), W - 1)];
#pragma unroll
    for (int k = 0; k < 5; ++k)                          // the five smallest in order
#pragma unroll
        for (int m = k + 1; m < 9; ++m)
            if (v[m] < v[k] || (v[k] != v[k] && v[m] == v[m])) {
                const float t = v[k];
                v[k] = v[m];
                v[m] = t;
            }
    out[i] = v[4];
}

// ---------------------------------------------------------------- semi-global aggregation
// One direction of _mvs.sgm: a warp per line of cells along the direction (lanes over the depth
// values of a cell), the cells of a line in the reference's scan order; the previous cell's
// values are read back from L. agg += L for every cell as the reference adds the directions.
__global__ void __launch_bounds__(128) sgm_dir_kernel(int D, int H, int W, int dy, int dx, float P1, float P2,
                                                      const float* __restrict__ cost, float* __restrict__ L,
                                                      float* __restrict__ agg, int first) {
    const int lane = threadIdx.x & 31;
    const int line = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const long long HW = (long long)H * W;
    // lines: dy == 0 -> rows; dx == 0 -> columns; diagonals -> cells with a common x*dy - y*dx
    int nlines, y, x, len;
    if (dy == 0) {
        nlines = H;
        if (line >= nlines) return;
        y = line;
        x = dx > 0 ? 0 : W - 1;
        len = W;
    } else if (dx == 0) {
        nlines = W;
        if (line >= nlines) return;
        x = line;
        y = dy > 0 ? 0 : H - 1;
        len = H;
    } else {
        nlines = H + W - 1;
        if (line >= nlines) return;
        // start cells: the first row (scan side) for lines that start there, then the first column
        const int ys = dy > 0 ? 0 : H - 1, xs = dx > 0 ? 0 : W - 1;
        if (line < W) {
            y = ys;
            x = dx > 0 ? line : W - 1 - line;
        } else {
            x = xs;
            y = dy > 0 ? line - W + 1 : H - 1 - (line - W + 1);
        }
        const int ny = dy > 0 ? H - y : y + 1, nx = dx > 0 ? W - x : x + 1;
        len = ny < nx ? ny : nx;
    }
    const unsigned full = 0xffffffffu;
    for (int s = 0; s < len; ++s, y += dy, x += dx) {
        const long long o = (long long)y * W + x;
        if (s == 0) {
            for (int d = lane; d < D; d += 32) L[d * HW + o] = cost[d * HW + o];
        } else {
            const long long po = o - (long long)dy * W - dx;
            float best = INFINITY;
            for (int d = lane; d < D; d += 32) best = fminf(best, L[d * HW + po]);
            for (int m = 16; m > 0; m >>= 1) best = fminf(best, __shfl_xor_sync(full, best, m));
            for (int d = lane; d < D; d += 32) {
                float v = L[d * HW + po];
                if (d > 0) {
                    const float a = __fadd_rn(L[(d - 1) * HW + po], P1);
                    if (a < v) v = a;
                }
                if (d < D - 1) {
                    const float b = __fadd_rn(L[(d + 1) * HW + po], P1);
                    if (b < v) v = b;
                }
                const float bp = __fadd_rn(best, P2);
                if (bp < v) v = bp;
                L[d * HW + o] = __fsub_rn(__fadd_rn(cost[d * HW + o], v), best);
            }
        }
        for (int d = lane; d < D; d += 32) {
            const float l = L[d * HW + o];
            agg[d * HW + o] = first ? __fadd_rn(0.f, l) : __fadd_rn(agg[d * HW + o], l);
        }
        __syncwarp();
    }
}

// All 8 directions in one launch, for D <= 32 M hypotheses: a warp per line, lane l keeps the values of
// hypotheses l M .. l M + M - 1 of the cell before in registers (their neighbours come from the next
// lanes), the cost of the cell after is on its way while this one is computed. The directions
// write volumes of their own, which sgm_sum_kernel adds in the reference's order. A direction at a
// time, each cell's values read back from global memory: 57 us a direction on 30 x 46 x 46 cells.
struct SgmDirs {
    int line0[9];                     // first line of each direction, then the total
};

template <int M>
__global__ void __launch_bounds__(128) sgm_lines_kernel(int D, int H, int W, const __grid_constant__ SgmDirs dirs, float P1,
                                                        float P2, const float* __restrict__ cost, float* __restrict__ L) {
    const int lane = threadIdx.x & 31;
    const int gl = (int)((blockIdx.x * 128 + threadIdx.x) >> 5);
    if (gl >= dirs.line0[8]) return;
    int k = 0;
    while (gl >= dirs.line0[k + 1]) ++k;
    const int line = gl - dirs.line0[k];
    // {0, 1}, {0, -1}, {1, 0}, {-1, 0}, {1, 1}, {1, -1}, {-1, 1}, {-1, -1}
    const int dy = k < 2 ? 0 : (k == 2 || k == 4 || k == 5 ? 1 : -1);
    const int dx = k < 2 ? (k == 0 ? 1 : -1) : (k < 4 ? 0 : (k == 4 || k == 6 ? 1 : -1));
    const long long HW = (long long)H * W;
    int y, x, len;
    if (dy == 0) {
        y = line;
        x = dx > 0 ? 0 : W - 1;
        len = W;
    } else if (dx == 0) {
        x = line;
        y = dy > 0 ? 0 : H - 1;
        len = H;
    } else {
        // start cells: the first row (scan side) for lines that start there, then the first column
        const int ys = dy > 0 ? 0 : H - 1, xs = dx > 0 ? 0 : W - 1;
        if (line < W) {
            y = ys;
            x = dx > 0 ? line : W - 1 - line;
        } else {
            x = xs;
            y = dy > 0 ? line - W + 1 : H - 1 - (line - W + 1);
        }
        const int ny = dy > 0 ? H - y : y + 1, nx = dx > 0 ? W - x : x + 1;
        len = ny < nx ? ny : nx;
    }
    const unsigned full = 0xffffffffu;
    float* out = L + (long long)k * D * HW;
    const int d0 = lane * M;
    long long o = (long long)y * W + x;
    const long long step = (long long)dy * W + dx;
    float prev[M], next[M];
    auto fetch = [&](long long at) {
#pragma unroll
        for (int m = 0; m < M; ++m) next[m] = d0 + m < D ? __ldg(cost + (d0 + m) * HW + at) : INFINITY;
    };
    fetch(o);
    for (int s = 0; s < len; ++s, o += step) {
        float cur[M];
#pragma unroll
        for (int m = 0; m < M; ++m) cur[m] = next[m];
        if (s + 1 < len) fetch(o + step);
        if (s > 0) {
            float best = INFINITY;
#pragma unroll
            for (int m = 0; m < M; ++m)
                if (d0 + m < D) best = fminf(best, prev[m]);
            for (int q = 16; q > 0; q >>= 1) best = fminf(best, __shfl_xor_sync(full, best, q));
            const float below = __shfl_up_sync(full, prev[M - 1], 1), above = __shfl_down_sync(full, prev[0], 1);
            const float bp = __fadd_rn(best, P2);
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int d = d0 + m;
                float v = prev[m];
                if (d > 0) {
                    const float a = __fadd_rn(m > 0 ? prev[m - 1 >= 0 ? m - 1 : 0] : below, P1);
                    if (a < v) v = a;
                }
                if (d < D - 1) {
                    const float b = __fadd_rn(m < M - 1 ? prev[m + 1 < M ? m + 1 : M - 1] : above, P1);
                    if (b < v) v = b;
                }
                if (bp < v) v = bp;
                cur[m] = __fsub_rn(__fadd_rn(cur[m], v), best);
            }
        }
        // (prev is read by the neighbouring lanes' shuffles above, so it changes only here)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            prev[m] = cur[m];
            if (d0 + m < D) out[(d0 + m) * HW + o] = cur[m];
        }
    }
}

__global__ void __launch_bounds__(256) sgm_sum_kernel(long long n, const float* __restrict__ L, float* __restrict__ agg) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) a = __fadd_rn(a, __ldg(L + k * n + i));
    agg[i] = a;
}

}  // namespace mvs

using namespace mvs;

extern "C" mvs_status mvs_sample_view(const mvs_sample_view_args* a, void* stream) {
    clear_error();
    if (!a) return fail(MVS_ERR_VALUE, "sample_view: null arguments");
    if (a->h < 1 || a->w < 1 || a->nch < 1 || a->D < 0 || a->H < 0 || a->W < 0)
        return fail(MVS_ERR_VALUE, "sample_view: bad shapes");
    const long long n = (long long)a->D * a->H * a->W;
    if (n == 0) return MVS_OK;
    if (!a->img || !a->cam || !a->Z || !a->out || !a->valid) return fail(MVS_ERR_VALUE, "sample_view: null pointer");
    SampleParams p;
    memset(&p, 0, sizeof(p));
    p.h = a->h; p.w = a->w; p.nch = a->nch; p.D = a->D; p.H = a->H; p.W = a->W;
    for (int k = 0; k < 9; ++k) p.R[k] = a->cam[k];
    for (int k = 0; k < 3; ++k) p.C[k] = a->cam[9 + k];
    p.f = a->cam[12]; p.k1 = a->cam[13]; p.k2 = a->cam[14]; p.k3 = a->cam[15]; p.cx = a->cam[16]; p.cy = a->cam[17];
    p.X0 = a->X0; p.Y0 = a->Y0; p.gsd = a->gsd;
    p.img = a->img; p.Z = a->Z; p.out = a->out; p.valid = a->valid;
    sample_view_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
    return check_launch("sample_view kernel");
}

extern "C" mvs_status mvs_box_sat_mean(int32_t B, int32_t H, int32_t W, const float* a, int32_t r, float* out,
                                       void* stream) {
    clear_error();
    if (r < 0) return fail(MVS_ERR_VALUE, "radius must be nonnegative");
    if (B < 0 || H < 0 || W < 0) return fail(MVS_ERR_VALUE, "box_sat_mean: negative shape");
    if ((long long)B * H * W == 0) return MVS_OK;
    if (!a || !out) return fail(MVS_ERR_VALUE, "box_sat_mean: null pointer");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const long long PH = H + 2LL * r + 1, PW = W + 2LL * r + 1;
    const size_t cs_bytes = sizeof(double) * (size_t)B * PH * W, sat_bytes = sizeof(double) * (size_t)B * PH * PW;
    void* ws = nullptr;
    MVS_CUDA(cudaMallocAsync(&ws, cs_bytes + sat_bytes, st), "box_sat_mean: scratch");
    double* cs = reinterpret_cast<double*>(ws);
    double* sat = cs + (size_t)B * PH * W;
    box_cols_kernel<<<(unsigned)(((long long)B * W + 127) / 128), 128, 0, st>>>(B, H, W, r, a, cs);
    mvs_status s = check_launch("box columns");
    if (s == MVS_OK) {
        box_rows_kernel<<<(unsigned)(((long long)B * PH + 127) / 128), 128, 0, st>>>(B, H, W, r, cs, sat);
        s = check_launch("box rows");
    }
    if (s == MVS_OK) {
        const long long n = (long long)B * H * W;
        box_mean_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(B, H, W, r, sat, out);
        s = check_launch("box mean");
    }
    cudaFreeAsync(ws, st);
    return s;
}

extern "C" mvs_status mvs_height_score(const mvs_height_score_args* a, void* stream) {
    clear_error();
    if (!a) return fail(MVS_ERR_VALUE, "height_score: null arguments");
    if (a->V < 2 || a->V > 16) return fail(MVS_ERR_VALUE, "height_score: %d views (2..16)", a->V);
    if (a->topk < 1 || a->topk > a->V) return fail(MVS_ERR_VALUE, "height_score: topk %d outside 1..%d", a->topk, a->V);
    const long long n = (long long)a->D * a->H * a->W;
    if (n == 0) return MVS_OK;
    if (!a->M || !a->S2 || !a->VA || !a->PP || !a->cxs || !a->cys || !a->cam_xy || !a->score)
        return fail(MVS_ERR_VALUE, "height_score: null pointer");
    ScoreParams p;
    memset(&p, 0, sizeof(p));
    p.V = a->V; p.D = a->D; p.H = a->H; p.W = a->W; p.topk = a->topk;
    p.full = (float)a->full; p.min_texture = (float)a->min_texture; p.full_texture = (float)a->full_texture;
    p.M = a->M; p.S2 = a->S2; p.VA = a->VA; p.PP = a->PP; p.cxs = a->cxs; p.cys = a->cys;
    for (int v = 0; v < a->V; ++v) {
        p.camx[v] = (float)a->cam_xy[2 * v];
        p.camy[v] = (float)a->cam_xy[2 * v + 1];
    }
    p.score = a->score; p.st = a->st; p.ref = a->ref;
    height_score_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
    return check_launch("height score kernel");
}

// Volumes of scratch that mvs_sgm keeps: one per direction, or one for the direction at a time when D
// is above 32 lanes' registers (or there is no room for eight).
static int sgm_volumes(int D) { return D <= 256 ? 8 : 1; }

extern "C" size_t mvs_sgm_scratch_bytes(int32_t D, int32_t H, int32_t W) {
    return D > 0 && H > 0 && W > 0 ? sizeof(float) * (size_t)sgm_volumes(D) * D * H * W : 0;
}

extern "C" mvs_status mvs_sgm_ws(int32_t D, int32_t H, int32_t W, const float* cost, float P1, float P2, float* agg,
                                 void* scratch, size_t scratch_bytes, void* stream) {
    clear_error();
    if (D < 0 || H < 0 || W < 0) return fail(MVS_ERR_VALUE, "sgm: negative shape");
    const long long n = (long long)D * H * W;
    if (n == 0) return MVS_OK;
    if (!cost || !agg) return fail(MVS_ERR_VALUE, "sgm: null pointer");
    if (!scratch || scratch_bytes < sizeof(float) * (size_t)n) return fail(MVS_ERR_VALUE, "sgm: scratch too small");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    float* L = reinterpret_cast<float*>(scratch);
    if (sgm_volumes(D) == 8 && scratch_bytes >= mvs_sgm_scratch_bytes(D, H, W)) {
        SgmDirs dirs;
        const int lines[8] = {H, H, W, W, H + W - 1, H + W - 1, H + W - 1, H + W - 1};
        dirs.line0[0] = 0;
        for (int k = 0; k < 8; ++k) dirs.line0[k + 1] = dirs.line0[k] + lines[k];
        const unsigned grid = (unsigned)(((long long)dirs.line0[8] * 32 + 127) / 128);
        if (D <= 32) sgm_lines_kernel<1><<<grid, 128, 0, st>>>(D, H, W, dirs, P1, P2, cost, L);
        else if (D <= 64) sgm_lines_kernel<2><<<grid, 128, 0, st>>>(D, H, W, dirs, P1, P2, cost, L);
        else if (D <= 128) sgm_lines_kernel<4><<<grid, 128, 0, st>>>(D, H, W, dirs, P1, P2, cost, L);
        else sgm_lines_kernel<8><<<grid, 128, 0, st>>>(D, H, W, dirs, P1, P2, cost, L);
        MVS_TRY(check_launch("sgm lines"));
        sgm_sum_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, L, agg);
        return check_launch("sgm sum");
    }
    static const int dirs[8][2] = {{0, 1}, {0, -1}, {1, 0}, {-1, 0}, {1, 1}, {1, -1}, {-1, 1}, {-1, -1}};
    for (int k = 0; k < 8; ++k) {
        const int dy = dirs[k][0], dx = dirs[k][1];
        const int nlines = dy == 0 ? H : (dx == 0 ? W : H + W - 1);
        const long long threads = (long long)nlines * 32;
        sgm_dir_kernel<<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(D, H, W, dy, dx, P1, P2, cost, L, agg,
                                                                          k == 0);
        MVS_TRY(check_launch("sgm direction"));
    }
    return MVS_OK;
}

extern "C" mvs_status mvs_sgm(int32_t D, int32_t H, int32_t W, const float* cost, float P1, float P2, float* agg,
                              void* stream) {
    clear_error();
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    size_t need = mvs_sgm_scratch_bytes(D, H, W);
    void* ws = nullptr;
    if (need && cost && agg) {
        cudaError_t e = cudaMallocAsync(&ws, need, st);
        if (e == cudaErrorMemoryAllocation && sgm_volumes(D) > 1) {   // no room: one direction at a time
            cudaGetLastError();
            need /= sgm_volumes(D);
            e = cudaMallocAsync(&ws, need, st);
        }
        MVS_CUDA(e, "sgm: scratch");
    }
    const mvs_status s = mvs_sgm_ws(D, H, W, cost, P1, P2, agg, ws, need, stream);
    if (ws) cudaFreeAsync(ws, st);
    return s;
}

// Scratch of mvs_height_eval: samples and window means.
struct EvalLayout {
    bool fused;
    int planes;
    size_t o_S, o_box, bytes;
};
static EvalLayout eval_layout(const mvs_height_eval_args* a) {
    EvalLayout l;
    const size_t n = (size_t)a->D * a->H * a->W;
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    l.planes = 3 * a->V + a->V * (a->V - 1) / 2;
    l.fused = a->W <= 1024 && height_box_smem(a->W, a->r) <= 200 * 1024;
    l.o_S = 0;
    l.o_box = l.o_S + up(n * a->V * 4);
    l.bytes = l.o_box + up(n * l.planes * 4);
    return l;
}

static mvs_status check_eval(const mvs_height_eval_args* a) {
    if (!a) return fail(MVS_ERR_VALUE, "height_eval: null arguments");
    if (a->V < 2 || a->V > 16) return fail(MVS_ERR_VALUE, "height_eval: %d views (2..16)", a->V);
    if (a->topk < 1 || a->topk > a->V) return fail(MVS_ERR_VALUE, "height_eval: topk %d outside 1..%d", a->topk, a->V);
    if (a->D < 0 || a->H < 0 || a->W < 0) return fail(MVS_ERR_VALUE, "height_eval: negative shape");
    if (a->D > 65535) return fail(MVS_ERR_UNSUPPORTED, "height_eval: %d hypotheses (at most 65535 per call)", a->D);
    if (a->r < 0) return fail(MVS_ERR_VALUE, "radius must be nonnegative");
    if ((long long)a->D * a->H * a->W == 0) return MVS_OK;
    if (!a->cams || !a->Z || !a->valid || !a->cxs || !a->cys || !a->score) return fail(MVS_ERR_VALUE, "height_eval: null pointer");
    for (int v = 0; v < a->V; ++v)
        if (!a->img[v] || a->img_h[v] < 1 || a->img_w[v] < 1) return fail(MVS_ERR_VALUE, "height_eval: bad image %d", v);
    if (!eval_layout(a).fused)
        return fail(MVS_ERR_UNSUPPORTED, "height_eval: a %d-column grid at radius %d does not fit in shared memory", a->W, a->r);
    return MVS_OK;
}

extern "C" size_t mvs_height_eval_scratch_bytes(const mvs_height_eval_args* a) {
    clear_error();
    if (check_eval(a) != MVS_OK) {
        clear_error();
        return 0;
    }
    return (long long)a->D * a->H * a->W == 0 ? 0 : eval_layout(a).bytes;
}

extern "C" mvs_status mvs_height_eval(const mvs_height_eval_args* a, void* scratch, size_t scratch_bytes, void* stream) {
    clear_error();
    MVS_TRY(check_eval(a));
    const long long n = (long long)a->D * a->H * a->W;
    if (n == 0) return MVS_OK;
    const EvalLayout l = eval_layout(a);
    if (!scratch || scratch_bytes < l.bytes)
        return fail(MVS_ERR_VALUE, "height_eval: scratch of %zu bytes below the %zu needed", scratch_bytes, l.bytes);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    char* ws = reinterpret_cast<char*>(scratch);
    EvalParams p;
    memset(&p, 0, sizeof(p));
    p.V = a->V; p.D = a->D; p.H = a->H; p.W = a->W;
    p.X0 = a->X0; p.Y0 = a->Y0; p.gsd = a->gsd;
    p.Z = a->Z;
    p.S = reinterpret_cast<float*>(ws + l.o_S);
    p.valid = a->valid;
    ScoreParams q;
    memset(&q, 0, sizeof(q));
    for (int v = 0; v < a->V; ++v) {
        const double* c = a->cams + 18 * v;
        EvalView& e = p.view[v];
        e.img = a->img[v];
        e.h = a->img_h[v];
        e.w = a->img_w[v];
        for (int k = 0; k < 9; ++k) e.R[k] = c[k];
        for (int k = 0; k < 3; ++k) e.C[k] = c[9 + k];
        e.f = c[12]; e.k1 = c[13]; e.k2 = c[14]; e.k3 = c[15]; e.cx = c[16]; e.cy = c[17];
        q.camx[v] = (float)c[9];
        q.camy[v] = (float)c[10];
    }
    height_sample_kernel<<<dim3((unsigned)((n + 255) / 256), a->V), 256, 0, st>>>(p);
    MVS_TRY(check_launch("height samples"));
    float* box = reinterpret_cast<float*>(ws + l.o_box);
    const size_t smem = height_box_smem(a->W, a->r);
    MVS_TRY(allow_smem(height_box_kernel, smem, "height box: shared memory attribute"));
    height_box_kernel<<<dim3(l.planes, a->D), 256, smem, st>>>(p, a->r, box);
    MVS_TRY(check_launch("height box"));
    q.V = a->V; q.D = a->D; q.H = a->H; q.W = a->W; q.topk = a->topk;
    q.full = (float)a->full; q.min_texture = (float)a->min_texture; q.full_texture = (float)a->full_texture;
    q.M = box;
    q.S2 = box + (long long)a->V * n;
    q.VA = box + 2LL * a->V * n;
    q.PP = box + 3LL * a->V * n;
    q.cxs = a->cxs; q.cys = a->cys;
    q.score = a->score; q.st = a->st; q.ref = a->ref;
    height_score_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(q);
    return check_launch("height score kernel");
}

extern "C" mvs_status mvs_height_stack(int32_t H, int32_t W, int32_t hc, int32_t wc, const float* Zc, int32_t K,
                                       const float* offs, float* up, float* stack, void* stream) {
    clear_error();
    if (H < 0 || W < 0 || K < 1 || hc < 1 || wc < 1) return fail(MVS_ERR_VALUE, "height_stack: bad shapes");
    if ((long long)H * W >= (1LL << 31)) return fail(MVS_ERR_VALUE, "height_stack: grid too large");
    if (H == 0 || W == 0) return MVS_OK;
    if (!Zc || !offs || !up || !stack) return fail(MVS_ERR_VALUE, "height_stack: null pointer");
    height_stack_kernel<<<(unsigned)(((long long)H * W + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        H, W, hc, wc, K, Zc, offs, up, stack);
    return check_launch("height stack");
}

extern "C" mvs_status mvs_height_pick(int32_t H, int32_t W, int32_t K, const float* score, const float* up,
                                      const float* offs, float weak, int32_t parabola, float cell, float* out,
                                      void* stream) {
    clear_error();
    if (H < 0 || W < 0 || K < 1) return fail(MVS_ERR_VALUE, "height_pick: bad shapes");
    if ((long long)H * W >= (1LL << 31)) return fail(MVS_ERR_VALUE, "height_pick: grid too large");
    if (H == 0 || W == 0) return MVS_OK;
    if (!score || !up || !offs || !out) return fail(MVS_ERR_VALUE, "height_pick: null pointer");
    const long long HW = (long long)H * W;
    height_pick_kernel<<<(unsigned)((HW + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        HW, K, score, up, offs, weak, parabola, cell, out);
    return check_launch("height pick");
}

extern "C" mvs_status mvs_median3(int32_t H, int32_t W, const float* a, float* out, void* stream) {
    clear_error();
    if (H < 0 || W < 0) return fail(MVS_ERR_VALUE, "median3: negative shape");
    if ((long long)H * W >= (1LL << 31)) return fail(MVS_ERR_VALUE, "median3: image too large");
    if (H == 0 || W == 0) return MVS_OK;
    if (!a || !out || a == out) return fail(MVS_ERR_VALUE, "median3: bad pointers");
    median3_kernel<<<(unsigned)(((long long)H * W + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        H, W, a, out);
    return check_launch("median3");
}
