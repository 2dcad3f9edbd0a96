// vc1cu_xform.cu - decoder-equivalent prediction of a motion field and the forward
// 8x8/8x4/4x8/4x4 transform + scalar quantiser of its residual.
//
// Prediction follows motion_compensate_mb / motion_compensate_4mv
// (encoder_motion_compensation.cpp:474-600). The transform is the reference's FP64 law
// (forward_transform_residual[_part], encoder_transform.cpp:797-1045): residual rows
// multiplied by the k8/k4 matrices in the reference's loop order, every product and sum
// rounded separately (this translation unit is compiled with --fmad=false and spells the
// operations with __dmul_rn/__dadd_rn), then scalar_quantize_level (:1067-1085).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>

#include "vc1cu_core.cuh"
#define VC1CU_ENT_TABLE __constant__ const
#include "vc1cu_entropy_lengths.h"
#include "vc1cu_pred.cuh"

namespace vc1cu {

// forward_transform::k4 / k8, forward_transform_tables.h:9-25 (inverse VC-1 basis)
__constant__ double c_k4[4][4] = {
    {0.0147058823529412, 0.0147058823529412, 0.0147058823529412, 0.0147058823529412},
    {0.0188356164383562, 0.0085616438356164, -0.0085616438356164, -0.0188356164383562},
    {0.0147058823529412, -0.0147058823529412, -0.0147058823529412, 0.0147058823529412},
    {0.0085616438356164, -0.0188356164383562, 0.0188356164383562, -0.0085616438356164}};
__constant__ double c_k8[8][8] = {
    {0.010416666667, 0.010416666667, 0.010416666667, 0.010416666667, 0.010416666667, 0.010416666667, 0.010416666667, 0.010416666667},
    {0.013840830450, 0.012975778547, 0.007785467128, 0.003460207612, -0.003460207612, -0.007785467128, -0.012975778547, -0.013840830450},
    {0.013698630137, 0.005136986301, -0.005136986301, -0.013698630137, -0.013698630137, -0.005136986301, 0.005136986301, 0.013698630137},
    {0.012975778547, -0.003460207612, -0.013840830450, -0.007785467128, 0.007785467128, 0.013840830450, 0.003460207612, -0.012975778547},
    {0.010416666667, -0.010416666667, -0.010416666667, 0.010416666667, 0.010416666667, -0.010416666667, -0.010416666667, 0.010416666667},
    {0.007785467128, -0.013840830450, 0.003460207612, 0.012975778547, -0.012975778547, -0.003460207612, 0.013840830450, -0.007785467128},
    {0.005136986301, -0.013698630137, 0.013698630137, -0.005136986301, -0.005136986301, 0.013698630137, -0.013698630137, 0.005136986301},
    {0.003460207612, -0.007785467128, 0.012975778547, -0.013840830450, 0.013840830450, -0.012975778547, 0.007785467128, -0.003460207612}};

// Vc1Encoder::chroma_mc_sample, encoder_motion_compensation.cpp:417-447 (P: future = false)
__device__ __forceinline__ int chroma_sample(const uint8_t* p, int pitch, int w, int h, int x, int y, int mvx, int mvy,
                                             int rnd) {
    int uvx = arshift(mvx + ((mvx & 3) == 3), 1);
    int uvy = arshift(mvy + ((mvy & 3) == 3), 1);
    if (uvx < 0) uvx += (uvx & 1); else uvx -= (uvx & 1);
    if (uvy < 0) uvy += (uvy & 1); else uvy -= (uvy & 1);
    const int ix = floor_div4(uvx), iy = floor_div4(uvy);
    const int fx = (uvx - ix * 4) * 2, fy = (uvy - iy * 4) * 2;
    const int sx = x + ix, sy = y + iy;
    auto S = [&](int xx, int yy) { return (int)__ldg(p + (size_t)iclamp(yy, 0, h - 1) * pitch + iclamp(xx, 0, w - 1)); };
    const int a = S(sx, sy);
    if (!fx && !fy) return a;
    const int b = S(sx + 1, sy), c = S(sx, sy + 1), d = S(sx + 1, sy + 1);
    const int value = a * (8 - fx) * (8 - fy) + b * fx * (8 - fy) + c * (8 - fx) * fy + d * fx * fy;
    return (value + (rnd ? 28 : 32)) >> 6;
}

__device__ __forceinline__ int median4(int a, int b, int c, int d) {
    if (a < b) {
        if (c < d) return (imin(b, d) + imax(a, c)) / 2;
        return (imin(b, c) + imax(a, d)) / 2;
    }
    if (c < d) return (imin(a, d) + imax(b, c)) / 2;
    return (imin(a, c) + imax(b, d)) / 2;
}

// One thread per luma pixel (and, for even pixels, the co-sited chroma pair).
__global__ void mc_kernel(const __grid_constant__ DevParams P, DevFrame ref, const int2* mvs, const int2* bmv,
                          const uint8_t* use4, int mode, uint8_t* dy, uint8_t* du, uint8_t* dv, int pitch_y, int pitch_c) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= P.W || y >= P.H) return;
    const int mx = x >> 4, my = y >> 4, pos = my * P.mbw + mx;
    const GlobSampler gs{ref.y, ref.pitch_y, P.W, P.H};
    int out[1];
    int2 cmv;
    if (use4[pos]) {
        const int k = ((y >> 3) & 1) * 2 + ((x >> 3) & 1);
        const int2 v = bmv[pos * 4 + k];
        predict_row<1>(gs, false, P.rnd, v.x, v.y, x, y, out);
        const int2 a = bmv[pos * 4 + 0], b = bmv[pos * 4 + 1], c = bmv[pos * 4 + 2], d = bmv[pos * 4 + 3];
        cmv = make_int2(median4(a.x, b.x, c.x, d.x), median4(a.y, b.y, c.y, d.y));
    } else {
        const int2 v = mvs[pos];
        predict_row<1>(gs, mode_bilinear(mode), P.rnd, v.x, v.y, x, y, out);
        cmv = v;
    }
    dy[(size_t)y * pitch_y + x] = (uint8_t)out[0];
    if (!(x & 1) && !(y & 1)) {
        const int cw = P.W / 2, ch = P.H / 2, cx = x >> 1, cy = y >> 1;
        if (cx < cw && cy < ch) {
            du[(size_t)cy * pitch_c + cx] = (uint8_t)chroma_sample(ref.u, ref.pitch_c, cw, ch, cx, cy, cmv.x, cmv.y, P.rnd);
            dv[(size_t)cy * pitch_c + cx] = (uint8_t)chroma_sample(ref.v, ref.pitch_c, cw, ch, cx, cy, cmv.x, cmv.y, P.rnd);
        }
    }
}

// Vc1Encoder::scalar_quantize_level, encoder_transform.cpp:1067-1085 (mquant = PQINDEX)
__device__ __forceinline__ int quantize_level(const DevParams& P, double coeff) {
    if (coeff == 0.0) return 0;
    const int sign = coeff < 0.0 ? -1 : 1;
    const double a = fabs(coeff);
    const double dq = (double)(2 * P.pq + (P.halfqp ? 1 : 0));
    const double offset = P.nonuniform ? (double)P.pq : 0.0;
    const int max_level = (1 << (P.pq < 8 ? 11 : 8)) - 1;
    int center = (int)llround(__ddiv_rn(__dsub_rn(a, offset), dq > 1.0 ? dq : 1.0));
    center = iclamp(center, 1, max_level);
    int best = 0;
    double besterr = __dmul_rn(a, a);
    for (int n = imax(1, center - 1); n <= imin(max_level, center + 1); ++n) {
        const double recon = __dadd_rn(__dmul_rn((double)n, dq), offset);
        const double e = __dsub_rn(a, recon);
        const double e2 = __dmul_rn(e, e);
        if (e2 < besterr) { besterr = e2; best = n; }
    }
    return sign * best;
}

// Threads per (MB, parent) of transform type t: one per partition row (partitions x rows).
__device__ __forceinline__ int xform_threads(int t) { return t == 1 || t == 2 ? 8 : 16; }

// One thread per (type, MB, parent, partition, transform row a): the row of the vertical stage
// and the outputs of frequency a (an 8x8 output column, transposed; a rectangle's row). Every
// product and sum is the reference's, in its order. Output layout [type][mb][parent][64].
__global__ void xform_kernel(const __grid_constant__ DevParams P, DevFrame src, DevFrame pred, int type_mask, double* coeffs,
                             int16_t* levels) {
    const int mbs = P.mbw * P.mbh;
    long off = (long)blockIdx.x * blockDim.x + threadIdx.x;
    int ti = -1, t = 0, nt = 0;
    for (int tt = 1; tt <= 4; ++tt) {
        if (!(type_mask & (1 << (tt - 1)))) continue;
        const long n = (long)mbs * 6 * xform_threads(tt);
        if (ti < 0) {
            if (off < n) {
                ti = nt;
                t = tt;
            } else {
                off -= n;
            }
        }
        ++nt;
    }
    if (ti < 0) return;
    const int per = xform_threads(t);
    const int sub = (int)(off % per);
    const long pk = off / per;
    const int k = (int)(pk % 6), mb = (int)(pk / 6);
    const int bh = (t == 2 || t == 4) ? 4 : 8, bw = (t == 3 || t == 4) ? 4 : 8;
    const int part = sub / bh, a = sub % bh;
    int ox = 0, oy = 0;
    if (t == 2) oy = part * 4;
    else if (t == 3) ox = part * 4;
    else if (t == 4) { ox = (part & 1) * 4; oy = (part >> 1) * 4; }
    const int mx = mb % P.mbw, my = mb / P.mbw;
    const bool chroma = k >= 4;
    const uint8_t* sp = chroma ? (k == 4 ? src.u : src.v) : src.y;
    const uint8_t* pp = chroma ? (k == 4 ? pred.u : pred.v) : pred.y;
    const int spitch = chroma ? src.pitch_c : src.pitch_y, ppitch = chroma ? pred.pitch_c : pred.pitch_y;
    const int w = chroma ? P.W / 2 : P.W, h = chroma ? P.H / 2 : P.H;
    const int bx = chroma ? mx : mx * 2 + (k & 1), by = chroma ? my : my * 2 + ((k >> 1) & 1);
    const int x0 = bx * 8 + ox, y0 = by * 8 + oy;
    const size_t base = (((size_t)ti * mbs + mb) * 6 + k) * 64;
    // output b of this thread's frequency a: transposed for 8x8, row-major for rectangles
    auto out_pos = [&](int b) {
        return (bw == 8 && bh == 8) ? base + (size_t)(oy + b) * 8 + ox + a : base + (size_t)(oy + a) * 8 + ox + b;
    };
    if (x0 >= w || y0 >= h || x0 + bw <= 0 || y0 + bh <= 0) {
        // a partition wholly outside the crop codes nothing (encoder_transform.cpp:1097)
        for (int b = 0; b < bw; ++b) {
            if (coeffs) coeffs[out_pos(b)] = 0.0;
            if (levels) levels[out_pos(b)] = 0;
        }
        return;
    }
    double trow[8];
    for (int x = 0; x < bw; ++x) {
        double acc = 0.0;
        for (int y = 0; y < bh; ++y) {
            const int sx = x0 + x, sy = y0 + y;
            const double r = (sx < 0 || sy < 0 || sx >= w || sy >= h)
                                 ? 0.0
                                 : (double)((int)__ldg(sp + (size_t)sy * spitch + sx) - (int)__ldg(pp + (size_t)sy * ppitch + sx));
            acc = __dadd_rn(acc, __dmul_rn(bh == 8 ? c_k8[a][y] : c_k4[a][y], r));
        }
        trow[x] = acc;
    }
    for (int b = 0; b < bw; ++b) {
        double acc = 0.0;
        for (int x = 0; x < bw; ++x) acc = __dadd_rn(acc, __dmul_rn(trow[x], bw == 8 ? c_k8[b][x] : c_k4[b][x]));
        const double c = __dmul_rn(1024.0, acc);
        if (coeffs) coeffs[out_pos(b)] = c;
        if (levels) levels[out_pos(b)] = (int16_t)quantize_level(P, c);
    }
}

// ---- inverse transform and reconstruction (encoder_transform.cpp:1058-1274, :1569-1585) ----

// Vc1Encoder::dequant_level at mquant = PQINDEX without DQUANT (2*PQ + HALFQP, plus PQ away from
// zero for the non-uniform quantiser)
__device__ __forceinline__ int dequant(const DevParams& P, int level) {
    if (!level) return 0;
    const int v = level * (2 * P.pq + (P.halfqp ? 1 : 0));
    return P.nonuniform ? v + (level > 0 ? P.pq : -P.pq) : v;
}

// The VC-1 8-point inverse butterfly (inverse_transform_8x8, :566-609); tail adds the second
// stage's +1 to the lower four outputs.
__device__ __forceinline__ void inv8(const int* s, int st, int* o, int ot, int bias, int shift, int tail) {
    int t1 = 12 * (s[0] + s[4 * st]) + bias, t2 = 12 * (s[0] - s[4 * st]) + bias;
    int t3 = 16 * s[2 * st] + 6 * s[6 * st], t4 = 6 * s[2 * st] - 16 * s[6 * st];
    const int t5 = t1 + t3, t6 = t2 + t4, t7 = t2 - t4, t8 = t1 - t3;
    t1 = 16 * s[st] + 15 * s[3 * st] + 9 * s[5 * st] + 4 * s[7 * st];
    t2 = 15 * s[st] - 4 * s[3 * st] - 16 * s[5 * st] - 9 * s[7 * st];
    t3 = 9 * s[st] - 16 * s[3 * st] + 4 * s[5 * st] + 15 * s[7 * st];
    t4 = 4 * s[st] - 9 * s[3 * st] + 15 * s[5 * st] - 16 * s[7 * st];
    o[0] = arshift(t5 + t1, shift);
    o[ot] = arshift(t6 + t2, shift);
    o[2 * ot] = arshift(t7 + t3, shift);
    o[3 * ot] = arshift(t8 + t4, shift);
    o[4 * ot] = arshift(t8 - t4 + tail, shift);
    o[5 * ot] = arshift(t7 - t3 + tail, shift);
    o[6 * ot] = arshift(t6 - t2 + tail, shift);
    o[7 * ot] = arshift(t5 - t1 + tail, shift);
}
// The 4-point one of the 8x4 / 4x8 / 4x4 partitions (inverse_partition, :1213-1272)
__device__ __forceinline__ void inv4(const int* s, int st, int* o, int ot, int bias, int shift) {
    const int t1 = 17 * (s[0] + s[2 * st]) + bias, t2 = 17 * (s[0] - s[2 * st]) + bias;
    const int t3 = 22 * s[st] + 10 * s[3 * st], t4 = 22 * s[3 * st] - 10 * s[st];
    o[0] = arshift(t1 + t3, shift);
    o[ot] = arshift(t2 - t4, shift);
    o[2 * ot] = arshift(t2 + t4, shift);
    o[3 * ot] = arshift(t1 - t3, shift);
}

// dequant_level (encoder_transform.cpp:1052-1065) at an MB's MQUANT: a DQUANT-derived MQUANT, or one
// other than PQINDEX, takes no HALFQP half step
__device__ __forceinline__ int dequant_mq(const DevParams& P, int level, int mquant, bool derived) {
    if (!level) return 0;
    const int v = level * (2 * mquant + ((!derived && mquant == P.pq && P.halfqp) ? 1 : 0));
    return P.nonuniform ? v + (level > 0 ? mquant : -mquant) : v;
}

// One thread per (MB, parent): every partition of the block's chosen type dequantised at PQINDEX
// or at the MB's MQUANT (mquant / derived: per-MB device arrays, or nullptr), inverse-transformed
// (with the DC-only shortcut of a partition whose only level is its DC) and added to the
// prediction with 8-bit clamping. tindex[t] is type t's index in the levels layout
// [type][mb][parent][64] (-1 for a type the layout does not hold).
__global__ void recon_kernel(const __grid_constant__ DevParams P, DevFrame pred, const int16_t* levels, int4 tindex,
                             const uint8_t* block_types, uint8_t* dy, uint8_t* du, uint8_t* dv, int pitch_y, int pitch_c,
                             const uint8_t* mquant, const uint8_t* derived) {
    const int mbs = P.mbw * P.mbh;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= mbs * 6) return;
    const int mb = idx / 6, k = idx - mb * 6, mx = mb % P.mbw, my = mb / P.mbw;
    const int t = block_types[idx];
    const int ti = t == 1 ? tindex.x : (t == 2 ? tindex.y : (t == 3 ? tindex.z : tindex.w));
    const int16_t* q64 = levels + (((size_t)ti * mbs + mb) * 6 + k) * 64;
    const int mq = mquant ? (int)mquant[mb] : P.pq;
    const bool der = derived && derived[mb];
    int res[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) res[i] = 0;
    const int np = t == 1 ? 1 : (t == 4 ? 4 : 2);
    for (int part = 0; part < np; ++part) {
        int ox = 0, oy = 0, bw = 8, bh = 8;
        if (t == 2) { bh = 4; oy = part * 4; }
        else if (t == 3) { bw = 4; ox = part * 4; }
        else if (t == 4) { bw = bh = 4; ox = (part & 1) * 4; oy = (part >> 1) * 4; }
        int a[64], tmp[64];
        int nonzero = 0, q0 = 0;
        for (int y = 0; y < 8; ++y)
            for (int x = 0; x < 8; ++x) {
                const int lv = (y < bh && x < bw) ? q64[(oy + y) * 8 + ox + x] : 0;
                nonzero += lv != 0;
                if (!y && !x) q0 = lv;
                a[y * 8 + x] = mquant ? dequant_mq(P, lv, mq, der) : dequant(P, lv);
                tmp[y * 8 + x] = 0;
            }
        if (nonzero == 1 && q0 != 0) {
            int dc = a[0];
            if (t == 1) { dc = arshift(3 * dc + 1, 1); dc = arshift(3 * dc + 16, 5); }
            else if (t == 2) { dc = arshift(3 * dc + 1, 1); dc = arshift(17 * dc + 64, 7); }
            else if (t == 3) { dc = arshift(17 * dc + 4, 3); dc = arshift(12 * dc + 64, 7); }
            else { dc = arshift(17 * dc + 4, 3); dc = arshift(17 * dc + 64, 7); }
            for (int y = 0; y < bh; ++y)
                for (int x = 0; x < bw; ++x) res[(oy + y) * 8 + ox + x] = dc;
            continue;
        }
        if (t == 1) {
            for (int col = 0; col < 8; ++col) inv8(a + col, 8, tmp + col * 8, 1, 4, 3, 0);
            for (int col = 0; col < 8; ++col) inv8(tmp + col, 8, a + col, 8, 64, 7, 1);
        } else if (t == 2) {
            for (int y = 0; y < 4; ++y) inv8(a + y * 8, 1, tmp + y * 8, 1, 4, 3, 0);
            for (int x = 0; x < 8; ++x) inv4(tmp + x, 8, a + x, 8, 64, 7);
        } else if (t == 3) {
            for (int y = 0; y < 8; ++y) inv4(a + y * 8, 1, tmp + y * 8, 1, 4, 3);
            for (int x = 0; x < 4; ++x) inv8(tmp + x, 8, a + x, 8, 64, 7, 1);
        } else {
            for (int y = 0; y < 4; ++y) inv4(a + y * 8, 1, tmp + y * 8, 1, 4, 3);
            for (int x = 0; x < 4; ++x) inv4(tmp + x, 8, a + x, 8, 64, 7);
        }
        for (int y = 0; y < bh; ++y)
            for (int x = 0; x < bw; ++x) res[(oy + y) * 8 + ox + x] = a[y * 8 + x];
    }
    const bool luma = k < 4;
    const int w = luma ? P.W : P.W / 2, h = luma ? P.H : P.H / 2;
    const int bx = luma ? mx * 2 + (k & 1) : mx, by = luma ? my * 2 + ((k >> 1) & 1) : my;
    const uint8_t* pp = luma ? pred.y : (k == 4 ? pred.u : pred.v);
    uint8_t* dp = luma ? dy : (k == 4 ? du : dv);
    const int pps = luma ? pred.pitch_y : pred.pitch_c, dps = luma ? pitch_y : pitch_c;
    for (int y = 0; y < 8 && by * 8 + y < h; ++y)
        for (int x = 0; x < 8 && bx * 8 + x < w; ++x) {
            const int v = pp[(size_t)(by * 8 + y) * pps + bx * 8 + x] + res[y * 8 + x];
            dp[(size_t)(by * 8 + y) * dps + bx * 8 + x] = (uint8_t)iclamp(v, 0, 255);
        }
}

void launch_recon(const DevParams& P, const DevFrame& pred, const int16_t* levels, int4 tindex, const uint8_t* block_types,
                  uint8_t* dy, uint8_t* du, uint8_t* dv, int pitch_y, int pitch_c, cudaStream_t s, const uint8_t* mquant,
                  const uint8_t* derived) {
    const int n = P.mbw * P.mbh * 6;
    recon_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(P, pred, levels, tindex, block_types, dy, du, dv, pitch_y, pitch_c,
                                                             mquant, derived);
}

// ---- transform type of the throughput preset (encoder_transform.cpp:1605-1712) ----------------

// One warp per MB: transform_metrics::scalar (transform_residual_metrics.h:29-61) with each lane
// summing half a row, then choose_transform_mb's candidate list and the preset's pick.
__global__ void fast_tt_kernel(const __grid_constant__ DevParams P, DevFrame src, DevFrame pred, uint8_t* types) {
    const int mb = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (mb >= P.mbw * P.mbh) return;
    const int mx = mb % P.mbw, my = mb / P.mbw;
    const int py = lane >> 1, px0 = (lane & 1) * 8;
    uint32_t sad = 0, hedge = 0, vedge = 0, grad = 0;
    const int y = my * 16 + py;
    if (y < P.H) {
        auto R = [&](int xx, int yy) {
            return (int)src.y[(size_t)yy * src.pitch_y + xx] - (int)pred.y[(size_t)yy * pred.pitch_y + xx];
        };
        for (int px = px0; px < px0 + 8 && mx * 16 + px < P.W; ++px) {
            const int x = mx * 16 + px;
            const int r = R(x, y);
            sad += (uint32_t)iabs(r);
            if ((py & 7) == 4) hedge += (uint32_t)iabs(r - R(x, y - 1));
            if ((px & 7) == 4) vedge += (uint32_t)iabs(r - R(x - 1, y));
            if (px > 0) grad += (uint32_t)iabs(r - R(x - 1, y));
            if (py > 0) grad += (uint32_t)iabs(r - R(x, y - 1));
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        sad += __shfl_xor_sync(0xffffffffu, sad, o);
        hedge += __shfl_xor_sync(0xffffffffu, hedge, o);
        vedge += __shfl_xor_sync(0xffffffffu, vedge, o);
        grad += __shfl_xor_sync(0xffffffffu, grad, o);
    }
    if (lane) return;
    const uint64_t S = sad, HE = hedge, VE = vedge, G = grad, lim = (uint64_t)(64 * P.pq);
    int list[4] = {1, 1, 1, 1}, count = 0;
    const bool split_x = mx == P.mbw - 1 && (P.W & 15) != 0, split_y = my == P.mbh - 1 && (P.H & 15) != 0;
    if (split_x && split_y) {
        list[count++] = 4;
    } else if (split_x || split_y) {
        list[count++] = split_x ? 3 : 2;
        if (S > lim && G > S * 2) list[count++] = 4;
    } else {
        list[count++] = 1;
        if (S > lim) {
            if (HE * 5 > VE * 6) list[count++] = 2;
            else if (VE * 5 > HE * 6) list[count++] = 3;
            else { list[count++] = 2; list[count++] = 3; }
            if (count < 4 && G > S * 2) list[count++] = 4;
        }
    }
    int chosen = list[0];
    if (count > 1) {
        int index = count - 1;
        if (list[index] == 4 && G * 2 <= S * 5) --index;
        chosen = list[index];
        if (chosen == 3 && index > 0 && list[index - 1] == 2 && HE >= VE) chosen = 2;
    }
    types[mb] = (uint8_t)chosen;
}

void launch_fast_tt(const DevParams& P, const DevFrame& src, const DevFrame& pred, uint8_t* types, cudaStream_t s) {
    const int mbs = P.mbw * P.mbh;
    fast_tt_kernel<<<(unsigned)((mbs + 3) / 4), 128, 0, s>>>(P, src, pred, types);
}

void launch_mc(const DevParams& P, const DevFrame& ref, const int2* mvs, const int2* bmv, const uint8_t* use4, int mode,
               uint8_t* dy, uint8_t* du, uint8_t* dv, int pitch_y, int pitch_c, cudaStream_t s) {
    dim3 grid((P.W + 127) / 128, P.H);
    mc_kernel<<<grid, 128, 0, s>>>(P, ref, mvs, bmv, use4, mode, dy, du, dv, pitch_y, pitch_c);
}

void launch_xform(const DevParams& P, const DevFrame& src, const DevFrame& pred, int type_mask, double* coeffs,
                  int16_t* levels, cudaStream_t s) {
    long n = 0;
    for (int t = 1; t <= 4; ++t)
        if (type_mask & (1 << (t - 1))) n += (long)P.mbw * P.mbh * 6 * (t == 1 || t == 2 ? 8 : 16);
    if (!n) return;
    xform_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(P, src, pred, type_mask, coeffs, levels);
}


// ---- transform RD of the default presets (choose_transform_mb, encoder_transform.cpp:1605-1780) ----
//
// One block of 128 threads per macroblock, its blocks, coefficients and levels in shared memory.
// Every stage spreads over the threads what is independent in it: one partition row per thread in
// the forward transforms, one coefficient in the quantiser, eight threads per parent block in the
// inverse transform, the SSE and the bit estimate, sixteen (32 at beam 8) per partition in the
// trellis. Every double operation is the reference's, in its order (this file is compiled without
// contraction); the statistics are integer sums. The work is latency (a trellis is a chain of up to
// 64 sorted steps) and FP64. With one lane per parent block and its arrays in local memory, a
// 1080p picture took 13.6 ms and the 32 sampled macroblocks of a mode decision 0.58 ms.

namespace {

// Dense rate tables built on the host from the VC-1 code lengths (vc1cu_entropy_lengths.h).
struct TrdTables {
    uint8_t ac_bits[8][2][64][64];  // direct AC code length (0: no direct code) [set][last][run][level]
    uint8_t max_level[8][2][64];    // max_direct_level
    int8_t max_run[8][2][64];       // max_direct_run (-1: none)
    // trellis_rate_bits: the family's least rate, [intra][PQINDEX < 8][last][run][level]. No set codes a
    // level of 127 or more but by Escape 3, so the last entry stands for every larger level.
    uint8_t family[2][2][2][64][128];
};

struct TrdArgs {
    DevParams P;
    DevFrame src, pred;
    const TrdTables* tab;
    const uint8_t* mquant;  // per MB, nullptr: PQINDEX
    vc1cu_trd_cfg cfg;
    double frame_mean;      // mean of the source luma plane (cached_luma_mean)
    vc1cu_tdecision* out;
    int16_t* levels;        // [mb][6][64] or nullptr
    const int* mb_list;     // nullptr: every MB; else entry i of out / levels is MB mb_list[i]
    int n_list;
};

__device__ __forceinline__ double dclamp(double v, double lo, double hi) { return v < lo ? lo : (hi < v ? hi : v); }
__device__ __forceinline__ double dmax(double a, double b) { return a < b ? b : a; }

// picture_double_quant (:1052-1056), dequant_level (:1058-1065), scalar_quantize_level (:1067-1085)
__device__ __forceinline__ int trd_double_quant(const DevParams& P, int mquant, bool derived) {
    return 2 * mquant + ((!derived && mquant == P.pq && P.halfqp) ? 1 : 0);
}
__device__ __forceinline__ int trd_max_level(const DevParams& P) { return (1 << (P.pq < 8 ? 11 : 8)) - 1; }
__device__ int trd_dequant(const DevParams& P, int level, int mquant, bool derived) {
    if (!level) return 0;
    long long v = (long long)level * trd_double_quant(P, mquant, derived);
    if (P.nonuniform) v += level > 0 ? mquant : -mquant;
    return (int)(v < INT_MIN ? INT_MIN : (v > INT_MAX ? INT_MAX : v));
}
__device__ int trd_squant(const DevParams& P, double coeff, int mquant, bool derived) {
    if (coeff == 0.0) return 0;
    const int sign = coeff < 0.0 ? -1 : 1;
    const double a = fabs(coeff);
    const double dq = (double)trd_double_quant(P, mquant, derived);
    const double offset = P.nonuniform ? (double)mquant : 0.0;
    const int max_level = trd_max_level(P);
    int center = (int)llround(__ddiv_rn(__dsub_rn(a, offset), dq > 1.0 ? dq : 1.0));
    center = iclamp(center, 1, max_level);
    int best = 0;
    double besterr = __dmul_rn(a, a);
    for (int n = imax(1, center - 1); n <= imin(max_level, center + 1); ++n) {
        const double e = __dsub_rn(a, __dadd_rn(__dmul_rn((double)n, dq), offset));
        const double e2 = __dmul_rn(e, e);
        if (e2 < besterr) { besterr = e2; best = n; }
    }
    return sign * best;
}

__device__ __forceinline__ void part_geometry(int t, int part, int& ox, int& oy, int& bw, int& bh) {
    ox = 0; oy = 0; bw = 8; bh = 8;
    if (t == 2) { bh = 4; oy = part * 4; }
    else if (t == 3) { bw = 4; ox = part * 4; }
    else if (t == 4) { bw = bh = 4; ox = (part & 1) * 4; oy = (part >> 1) * 4; }
}
__device__ __forceinline__ int part_count(int t) { return t == 1 ? 1 : (t == 4 ? 4 : 2); }

// ---- the perceptual lambda scale (perceptual_lambda_scale, encoder_aq.cpp:405-653) ----------

// The G neighbouring lanes that share one task; lane: this thread's place among them.
struct Team {
    unsigned mask;
    int lane, size;
    __device__ __forceinline__ uint32_t sum(uint32_t v) const { return __reduce_add_sync(mask, v); }
    __device__ __forceinline__ int low(int v) const { return __reduce_min_sync(mask, v); }
    __device__ __forceinline__ int high(int v) const { return __reduce_max_sync(mask, v); }
};

struct AqStats {
    double mean = 128.0, grad_avg = 0.0, residual_avg = 0.0;
    int mn = 255, mx = 0, edges = 0, n = 0;
    uint32_t dark_grad = 0;  // the gradients of samples in [2, 112] (luma blocks)
    int dark_n = 0;
};

__device__ AqStats aq_stats(const Team& g, const uint8_t* plane, int pitch, int pw, int ph, int sx, int sy, int sw, int sh,
                            const uint8_t* pp, int ppitch) {
    AqStats st;
    uint32_t sum = 0, grad = 0, residual = 0, dark = 0;
    int grad_n = 0, n = 0, edges = 0, dark_n = 0, mn = 255, mx = 0;
    const int cw = imin(sw, pw - sx), chh = imin(sh, ph - sy);
    for (int i = g.lane; i < sw * sh; i += g.size) {
        const int x = i % sw, y = i / sw;
        if (x >= cw || y >= chh) continue;
        const uint8_t* at = plane + (size_t)(sy + y) * pitch + sx + x;
        const int v = __ldg(at);
        sum += (uint32_t)v;
        mn = imin(mn, v);
        mx = imax(mx, v);
        ++n;
        if (pp) residual += (uint32_t)iabs(v - (int)__ldg(pp + (size_t)(sy + y) * ppitch + sx + x));
        const bool dk = v >= 2 && v <= 112;
        auto edge = [&](int d) {
            grad += (uint32_t)d;
            ++grad_n;
            if (d >= 96) ++edges;
            if (dk) {
                dark += (uint32_t)d;
                ++dark_n;
            }
        };
        if (x > 0) edge(iabs(v - (int)__ldg(at - 1)));
        if (y > 0) edge(iabs(v - (int)__ldg(at - pitch)));
    }
    sum = g.sum(sum);
    grad = g.sum(grad);
    grad_n = (int)g.sum((uint32_t)grad_n);
    st.n = (int)g.sum((uint32_t)n);
    st.edges = (int)g.sum((uint32_t)edges);
    st.dark_grad = g.sum(dark);
    st.dark_n = (int)g.sum((uint32_t)dark_n);
    st.mn = g.low(mn);
    st.mx = g.high(mx);
    if (pp) residual = g.sum(residual);
    if (st.n) {
        st.mean = (double)sum / st.n;
        st.grad_avg = (double)grad / imax(1, grad_n);
        st.residual_avg = pp ? (double)residual / st.n : 0.0;
    }
    return st;
}

__device__ __forceinline__ double aq_activity(const AqStats& st) {
    const double range = (double)imax(0, st.mx - st.mn);
    const double g = dclamp((st.grad_avg - 0.35) / 5.0, 0.0, 1.0);
    const double r = dclamp((range - 1.5) / 18.0, 0.0, 1.0);
    return dmax(g, r);
}

// plane (pitch) of w x h; pp the prediction (or nullptr); luma: the picture's luma plane when the
// block is chroma (the luma context), else nullptr
// adjacency_out (luma blocks): the quiet-block-next-to-detail term, 0 when the scale is not
// computed (perceptual_lambda_scale's adjacency_out, encoder_aq.cpp:410, :641)
// The team's threads all call it and all get the result.
__device__ double aq_scale(const Team& g, const TrdArgs& A, const uint8_t* plane, int pitch, int w, int h, int x0, int y0,
                           int bw, int bh, const uint8_t* pp, int ppitch, const uint8_t* luma, int lpitch, double* adjacency_out = nullptr) {
    const vc1cu_trd_cfg& c = A.cfg;
    if (adjacency_out) *adjacency_out = 0.0;
    if (!c.adaptive_quality || c.aq_strength <= 0.0) return 1.0;
    const AqStats st = aq_stats(g, plane, pitch, w, h, x0, y0, bw, bh, pp, ppitch);
    if (!st.n) return 1.0;
    const double range = (double)imax(0, st.mx - st.mn);
    const double contrast = dclamp((range - 64.0) / 144.0, 0.0, 1.0) * dclamp((st.grad_avg - 7.0) / 40.0, 0.0, 1.0);
    const double edge_density = dclamp((double)st.edges / imax(1, st.n / 3), 0.0, 1.0);
    const double motion = dclamp((st.residual_avg - 5.0) / 30.0, 0.0, 1.0);
    if (luma) {
        const AqStats ly = aq_stats(g, luma, lpitch, A.P.W, A.P.H, x0 * 2, y0 * 2, bw * 2, bh * 2, nullptr, 0);
        const double chroma_detail =
            dmax(dclamp((st.grad_avg - 1.5) / 11.0, 0.0, 1.0), dclamp((range - 6.0) / 48.0, 0.0, 1.0));
        const double luma_activity = aq_activity(ly);
        const double luma_flat = dclamp((0.42 - luma_activity) / 0.42, 0.0, 1.0);
        const double luma_visibility = 0.20 + 0.80 * dclamp((ly.mean - 1.0) / 14.0, 0.0, 1.0);
        const double chroma_on_flat = luma_flat * chroma_detail * luma_visibility;
        const double frame_mean = A.frame_mean;
        const double dim_area = dclamp((132.0 - ly.mean) / 104.0, 0.0, 1.0);
        const double dim_frame = dclamp((132.0 - frame_mean) / 104.0, 0.0, 1.0);
        const double not_black = dclamp((ly.mean - 0.75) / 9.0, 0.0, 1.0);
        const double dim_detail = dmax(dim_area, 0.80 * dim_frame) * not_black * chroma_detail;
        const double protect = c.aq_strength * (1.90 * chroma_on_flat + 0.70 * dim_detail + 0.12 * contrast +
                                                0.08 * edge_density + 0.05 * motion);
        return dclamp(1.0 / (1.0 + protect), 0.24, 1.0);
    }
    const double dark_avg = st.dark_n ? (double)st.dark_grad / st.dark_n : 0.0;
    const double dark_window = dclamp((118.0 - st.mean) / 96.0, 0.0, 1.0) * dclamp((st.mean - 1.0) / 13.0, 0.0, 1.0);
    const double dark_detail = dark_window * dclamp(dark_avg / 10.0, 0.0, 1.0);
    const double frame_mean = (w == A.P.W && h == A.P.H) ? A.frame_mean : st.mean;
    const double dim_area = dclamp((142.0 - st.mean) / 116.0, 0.0, 1.0);
    const double dim_frame = dclamp((142.0 - frame_mean) / 116.0, 0.0, 1.0);
    const double not_black = dclamp((st.mean - 0.75) / 9.0, 0.0, 1.0);
    const double dim_detail = dmax(dim_area, 0.82 * dim_frame) * not_black * aq_activity(st);
    const int pad = 4;
    const int cx0 = imax(0, x0 - pad), cy0 = imax(0, y0 - pad);
    const int cx1 = imin(w, x0 + bw + pad), cy1 = imin(h, y0 + bh + pad);
    uint32_t ring_grad = 0;
    int ring_n = 0, ring_edges = 0;
    const int rw = cx1 - cx0, rh = cy1 - cy0;
    for (int i = g.lane; i < rw * rh; i += g.size) {
        const int px = cx0 + i % rw, py = cy0 + i / rw;
        if (px >= x0 && px < x0 + bw && py >= y0 && py < y0 + bh) continue;
        const uint8_t* at = plane + (size_t)py * pitch + px;
        const int v = __ldg(at);
        if (px > cx0) {
            const int d = iabs(v - (int)__ldg(at - 1));
            ring_grad += (uint32_t)d;
            if (d >= 64) ++ring_edges;
            ++ring_n;
        }
        if (py > cy0) {
            const int d = iabs(v - (int)__ldg(at - pitch));
            ring_grad += (uint32_t)d;
            if (d >= 64) ++ring_edges;
            ++ring_n;
        }
    }
    ring_grad = g.sum(ring_grad);
    ring_n = (int)g.sum((uint32_t)ring_n);
    ring_edges = (int)g.sum((uint32_t)ring_edges);
    const double ring_grad_avg = ring_n ? (double)ring_grad / ring_n : 0.0;
    const double ring_edge_density = ring_n ? (double)ring_edges / ring_n : 0.0;
    const double context_activity = dclamp((ring_grad_avg - 10.0) / 36.0, 0.0, 1.0) +
                                    0.8 * dclamp((ring_edge_density - 0.04) / 0.24, 0.0, 1.0);
    const double quietness = dclamp((18.0 - st.grad_avg) / 14.0, 0.0, 1.0);
    const double neutral_window = dclamp((190.0 - st.mean) / 120.0, 0.0, 1.0) * dclamp((st.mean - 6.0) / 30.0, 0.0, 1.0);
    const double adjacency = quietness * neutral_window * dclamp(context_activity, 0.0, 1.5);
    if (adjacency_out) *adjacency_out = adjacency;
    double bright_field_detail = 0.0;
    if ((contrast > 0.15 || edge_density > 0.25) && w == A.P.W && h == A.P.H) {
        const double bright_field = dclamp((frame_mean - 165.0) / 55.0, 0.0, 1.0);
        bright_field_detail = bright_field * dmax(contrast, 0.65 * edge_density);
    }
    const double protect = c.aq_strength * (8.50 * dark_detail + 1.45 * dim_detail + 0.20 * contrast + 0.10 * edge_density +
                                            0.08 * motion + 1.00 * adjacency + 2.00 * bright_field_detail);
    return dclamp(1.0 / (1.0 + protect), 0.18, 1.0);
}

// ---- bit estimates (encoder_entropy.cpp:182-302, encoder_transform.cpp:1344-1553) ---------

__device__ __forceinline__ int ac_direct(const TrdTables* T, int set, int run, int level, bool last) {
    if (run < 0 || run > 63 || level < 0 || level >= 64) return 0;
    return __ldg(&T->ac_bits[set][last ? 1 : 0][run][level]);
}
__device__ __forceinline__ int ac_max_level(const TrdTables* T, int set, int run, bool last) {
    if (run < 0 || run > 63) return 0;
    return __ldg(&T->max_level[set][last ? 1 : 0][run]);
}
__device__ __forceinline__ int ac_max_run(const TrdTables* T, int set, int level, bool last) {
    if (level < 0 || level >= 64) return -1;
    return __ldg(&T->max_run[set][last ? 1 : 0][level]);
}
__device__ __forceinline__ int esc3_level_bits(const DevParams& P) { return P.pq < 8 ? 11 : 8; }

// The length of one coefficient as write_ac_coeff (encoder_entropy.cpp:246-302) codes it, as a
// function of the Escape-3 length header's state: the length where Escape 3 is not taken (0: it is,
// whatever the state), and Escape 3's without the header. Escape 3 is taken when it is the shorter,
// the header counted until one was written.
struct CoeffBits {
    int other, esc3;
};
__device__ CoeffBits ac_coeff_bits(const TrdArgs& A, int run, int level, bool last) {
    const DevParams& P = A.P;
    const int set = A.cfg.coding_set, mag = iabs(level), esc = ent::kAcEscapeBits[set];
    CoeffBits r{0, esc + 2 + 1 + 6 + 1 + esc3_level_bits(P)};
    if (!A.cfg.use_vlc) return r;
    if (const int d = ac_direct(A.tab, set, run, mag, last)) {
        r.other = d + 1;
        r.esc3 = 1000000;  // a direct code is always taken
        return r;
    }
    const int level_delta = ac_max_level(A.tab, set, run, last);
    if (set != 3 && level_delta > 0 && mag > level_delta) {
        if (const int b = ac_direct(A.tab, set, run, mag - level_delta, last)) r.other = esc + 1 + b + 1;
    }
    const int run_delta = ac_max_run(A.tab, set, mag, last);
    if (run_delta >= 0 && run > run_delta) {
        if (const int b = ac_direct(A.tab, set, run - run_delta - 1, mag, last)) {
            const int bits = esc + 2 + b + 1;
            if (!r.other || bits < r.other) r.other = bits;
        }
    }
    return r;
}

__device__ __forceinline__ const uint8_t* inter_scan(int t, int& n) {
    if (t == 1) { n = 64; return ent::kInterScan; }
    if (t == 2) { n = 32; return ent::kInterScan8x4; }
    if (t == 3) { n = 32; return ent::kInterScan4x8; }
    n = 16;
    return ent::kInterScan4x4;
}

__device__ __forceinline__ int tt_table(const DevParams& P) { return P.pq <= 4 ? 0 : (P.pq <= 12 ? 1 : 2); }
__device__ __forceinline__ int subblkpat_bits(const DevParams& P, int skip) { return ent::kSubblkBits[tt_table(P)][14 - skip]; }
__device__ __forceinline__ int rect_subblkpat_bits(int skip) { return skip == 0 ? 1 : 2; }  // decode012 of 0 / 2 / 1
__device__ int ttblk_bits(const DevParams& P, int t, int skip) {
    int variant;
    if (t == 1) variant = 0;
    else if (t == 4) variant = 7;
    else if (t == 2) variant = skip == 0 ? 1 : (skip == 1 ? 2 : 3);
    else variant = skip == 0 ? 4 : (skip == 1 ? 5 : 6);
    const int tab = tt_table(P);
    int symbol = 0;
    for (int s = 0; s < 8; ++s)
        if (ent::kTtSymbolVariant[tab][s] == variant) { symbol = s; break; }
    return ent::kTtblkBits[tab][symbol];
}
__device__ int ttmb_macro_bits(const DevParams& P, int t, int first_skip) {
    int symbol = 8;
    if (t == 2) symbol = first_skip == 1 ? 10 : (first_skip == 2 ? 9 : 11);
    else if (t == 3) symbol = first_skip == 1 ? 13 : (first_skip == 2 ? 12 : 14);
    else if (t == 4) symbol = 15;
    return ent::kTtmbBits[tt_table(P)][symbol];
}
__device__ int ttmb_block_bits(const DevParams& P, int t, int first_skip) {
    int value;
    if (t == 1) value = 0;
    else if (t == 4) value = 7;
    else if (t == 2) value = first_skip == 0 ? 3 : (first_skip == 1 ? 2 : 1);
    else value = first_skip == 0 ? 6 : (first_skip == 1 ? 5 : 4);
    return ent::kTtmbBits[tt_table(P)][value];
}

// A TransformParentDecision in shared memory
struct TParent {
    int16_t q[64];      // the partitions' levels in their sub-rectangles of the 8x8 grid
    double distortion;
    uint32_t bits;      // estimate_parent_payload_bits
    // the coefficients' bits alone: coded before any Escape-3 length header was written (esc0: one is
    // written among them), and after
    uint32_t coef0, coef1;
    uint8_t type, skip, esc0;
};

// estimate_ttblk_bits (:1545-1553)
__device__ uint32_t parent_ttblk_bits(const DevParams& P, const TParent& p) {
    const int np = part_count(p.type);
    if (p.skip == (1 << np) - 1) return 0;
    int bits = ttblk_bits(P, p.type, p.skip);
    if (p.type == 4) bits += subblkpat_bits(P, p.skip);
    return (uint32_t)bits;
}

// The grid index of partition `part`'s first coefficient, and the grid positions it covers.
__device__ __forceinline__ int part_origin(int t, int part) {
    return t == 2 ? 32 * part : (t == 3 ? 4 * part : (t == 4 ? 32 * (part >> 1) + 4 * (part & 1) : 0));
}
__device__ __forceinline__ uint64_t part_cells(int t, int part) {
    return (t == 1 ? ~0ull : t == 2 ? 0xFFFFFFFFull : t == 3 ? 0x0F0F0F0F0F0F0F0Full : 0x0F0F0F0Full) << part_origin(t, part);
}

// ---- the forward transform (forward_transform_residual_part, :935-1045) -------------------------

// One partition row of a block's residual (px: source minus prediction, zero outside the raster):
// the vertical stage of row `a` and the outputs of its frequency, into the 8x8 grid c (8x8 output
// transposed, rectangles row-major in their place).
__device__ __forceinline__ void forward_row(const int16_t* px, int t, int part, int a, double* c) {
    const int bh = (t == 2 || t == 4) ? 4 : 8, bw = (t == 3 || t == 4) ? 4 : 8, org = part_origin(t, part);
    double row[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        double acc = 0.0;
        if (x < bw)
            for (int y = 0; y < bh; ++y)
                acc = __dadd_rn(acc, __dmul_rn(bh == 8 ? c_k8[a][y] : c_k4[a][y], (double)px[org + y * 8 + x]));
        row[x] = acc;
    }
    for (int b = 0; b < bw; ++b) {
        double acc = 0.0;
#pragma unroll
        for (int x = 0; x < 8; ++x)
            if (x < bw) acc = __dadd_rn(acc, __dmul_rn(row[x], bw == 8 ? c_k8[b][x] : c_k4[b][x]));
        c[(t == 1 ? b * 8 + a : org + a * 8 + b)] = __dmul_rn(1024.0, acc);
    }
}

// ---- trellis_quantize (:1873-2088) ---------------------------------------------------------

// trellis_coeff_weight (:1859-1871)
__device__ __forceinline__ double trellis_weight(int t, int index) {
    const int row = index >> 3, col = index & 7;
    auto e8 = [](int i) { return (i & 3) == 0 ? 1152.0 : ((i & 3) == 2 ? 1168.0 : 1156.0); };
    auto e4 = [](int i) { return (i & 1) ? 1168.0 : 1156.0; };
    const double ex = (t == 3 || t == 4) ? e4(col) : e8(col), ey = (t == 2 || t == 4) ? e4(row) : e8(row);
    return (ex * ey) / (1024.0 * 1024.0);
}

constexpr int kTrdThreads = 128;

// One trellis's working memory: the successors of a step, the surviving states and, per scan
// position, the state each survivor extends and the candidate it took there.
template <int BEAM>
struct TrellisMem {
    static constexpr int kTeam = 4 * BEAM;  // four candidate lanes per state
    uint64_t score[kTeam];
    double dist[kTeam];
    double sdist[BEAM];
    uint32_t bits[kTeam], aux[kTeam], sbits[BEAM], saux[BEAM];
    uint8_t bp[64 * BEAM];
};
constexpr int kTrellisBytes = (kTrdThreads / 16) * (int)sizeof(TrellisMem<4>);
static_assert((kTrdThreads / 32) * (int)sizeof(TrellisMem<8>) <= kTrellisBytes + 1024, "trellis memory");

// Candidate ci of a position whose scalar level is q0: 0, q0, one nearer zero, one farther (kept within
// max_level); a candidate that repeats an earlier one, or that the search does not try, is absent.
__device__ __forceinline__ int trellis_candidate(int q0, int ci, bool wide, int max_level, bool& present) {
    const int sign = q0 > 0 ? 1 : -1;
    const int v = ci == 0 ? 0 : (ci == 1 ? q0 : (ci == 2 ? q0 - sign : iclamp(q0 + sign, -max_level, max_level)));
    present = ci == 0 || (q0 != 0 && (ci == 1 || (ci == 2 ? v != 0 : (wide && v != q0))));
    return v;
}

// Levels q of one partition's coefficients c (both at the partition's origin in the 8x8 grid), given
// the scalar levels, along scan[0..n): positions first_scan.. (1 for intra blocks, whose DC is coded
// apart), with the rates of the intra or inter family. A team of 4 x BEAM lanes: lane = state * 4 +
// candidate computes one successor; survivors are the least of (score, bits, distortion), equal ones in
// the order the reference makes them, found by ranking every successor against every other. A
// position whose scalar level is zero has one successor per state and mostly keeps their order, which
// costs one comparison with the next state instead. A survivor's exact rate (its last coefficient
// coded as last) follows from the rate it carries and that coefficient's run and level.
template <int BEAM>
__device__ void trellis_team(const Team& g, const TrdArgs& A, const double* c, const int16_t* scalar, int t, double lambda_scale,
                             int mquant, const uint8_t* scan, int n, int first_scan, bool intra, int16_t* q,
                             TrellisMem<BEAM>& mem) {
    constexpr int G = TrellisMem<BEAM>::kTeam;
    const DevParams& P = A.P;
    const bool derived = mquant != P.pq, wide = A.cfg.trellis >= 2;
    const double qscale = (double)trd_double_quant(P, mquant, derived);
    const int max_level = trd_max_level(P);
    const double lambda = 0.15 * qscale * qscale * dclamp(lambda_scale, 0.20, 1.50);
    const uint8_t(*fam)[64][128] = A.tab->family[intra ? 1 : 0][P.pq < 8 ? 1 : 0];
    const int si = g.lane >> 2, ci = g.lane & 3;
    int count = 1;
    // the lane's state: aux = last position + 1 | run << 8 | level << 16 (clamped) | 1 << 24 of its last coefficient
    double dist = 0.0;
    uint32_t bits = 0, aux = (uint32_t)first_scan;
    for (int s = first_scan; s < n; ++s) {
        const int idx = scan[s];
        const int q0 = scalar[idx];
        bool present;
        const int level = trellis_candidate(q0, q0 ? ci : 0, wide, max_level, present);
        const double e = c[idx] - (double)trd_dequant(P, level, mquant, derived);
        const double nd = dist + e * e * trellis_weight(t, idx);
        uint32_t nb = bits, na = aux;
        if (level != 0) {
            const int run = s - (int)(aux & 255), mag = imin(iabs(level), 127);
            nb += __ldg(&fam[0][run][mag]);
            na = (uint32_t)(s + 1) | ((uint32_t)run << 8) | ((uint32_t)mag << 16) | (1u << 24);
        }
        const uint64_t score = (uint64_t)__double_as_longlong(nd + lambda * (double)nb);  // >= 0: ordered as integers
        if (q0 == 0) {
            const uint64_t ns = __shfl_down_sync(g.mask, score, 4, G);
            const uint32_t nnb = __shfl_down_sync(g.mask, nb, 4, G);
            const double nnd = __shfl_down_sync(g.mask, nd, 4, G);
            const bool moves = si + 1 < count && (ns < score || (ns == score && (nnb < nb || (nnb == nb && nnd < nd))));
            if (!__any_sync(g.mask, moves)) {
                dist = nd;
                if (ci == 0 && si < count) mem.bp[s * BEAM + si] = (uint8_t)(si << 2);
                continue;
            }
        }
        const bool valid = si < count && present && (q0 != 0 || ci == 0);
        mem.score[g.lane] = valid ? score : ~0ull;
        mem.dist[g.lane] = nd;
        mem.bits[g.lane] = nb;
        mem.aux[g.lane] = na;
        const int made = __popc(__ballot_sync(g.mask, valid) & g.mask);
        __syncwarp(g.mask);
        int rank = 0;
#pragma unroll 4
        for (int j = 0; j < G; ++j) {
            const uint64_t sj = mem.score[j];
            bool less = sj < score;
            if (sj == score && j != g.lane) {
                const uint32_t bj = mem.bits[j];
                const double dj = mem.dist[j];
                less = bj != nb ? bj < nb : (dj != nd ? dj < nd : j < g.lane);
            }
            rank += less ? 1 : 0;
        }
        if (valid && rank < BEAM) {
            mem.sdist[rank] = nd;
            mem.sbits[rank] = nb;
            mem.saux[rank] = na;
            mem.bp[s * BEAM + rank] = (uint8_t)((si << 2) | ci);
        }
        __syncwarp(g.mask);
        count = imin(made, BEAM);
        if (si < count) {
            dist = mem.sdist[si];
            bits = mem.sbits[si];
            aux = mem.saux[si];
        }
    }
    // the exact rate of each survivor, then the least D + lambda R, the first of equal ones
    uint32_t exact = bits;
    if (aux >> 24) {
        const int run = (int)((aux >> 8) & 255), mag = (int)((aux >> 16) & 255);
        exact = bits - __ldg(&fam[0][run][mag]) + __ldg(&fam[1][run][mag]);
    }
    if (ci == 0) mem.score[si] = (uint64_t)__double_as_longlong(dist + lambda * (double)exact);
    __syncwarp(g.mask);
    if (g.lane == 0) {
        int best = 0;
        for (int i = 1; i < count; ++i)
            if (mem.score[i] < mem.score[best]) best = i;
        int j = best;
        for (int s = n - 1; s >= first_scan; --s) {
            const int code = mem.bp[s * BEAM + j], idx = scan[s];
            bool present;
            q[idx] = (int16_t)trellis_candidate(scalar[idx], code & 3, wide, max_level, present);
            j = code >> 2;
        }
    }
    __syncwarp(g.mask);
}

// One macroblock's blocks and the search's working set.
struct TrdShared {
    double c[24][64];              // coefficients of (candidate type, parent)
    alignas(16) uint8_t trellis[kTrellisBytes + 1024];
    TParent pool[36];              // 24 candidate parents, 6 trellis macro parents, 6 trellis block parents
    int16_t sq[24][64];            // scalar levels of (candidate type, parent)
    int tmp[kTrdThreads / 8][64];  // the inverse transforms' first stage, one parent per eight threads
    int16_t px[6][64];             // residual, zero outside the raster
    uint8_t src[6][64], pred[6][64];
    double lscale;                 // the macroblock's perceptual lambda scale
    int list[4], count;            // candidate types
    uint8_t need[6], macro_type;   // the block winners' types, the macroblock winner's
    uint8_t jobs[48];              // trellis partitions: job * 4 + partition
    int n_jobs;
    int chosen[6];
};

// Visible columns / rows of block k.
__device__ __forceinline__ int2 block_extent(const DevParams& P, int mx, int my, int k) {
    const bool chroma = k >= 4;
    const int x0 = (chroma ? mx : mx * 2 + (k & 1)) * 8, y0 = (chroma ? my : my * 2 + ((k >> 1) & 1)) * 8;
    return make_int2(iclamp((chroma ? P.W / 2 : P.W) - x0, 0, 8), iclamp((chroma ? P.H / 2 : P.H) - y0, 0, 8));
}

// The rest of evaluate_transform_parent (:1555-1590) of a parent whose levels are in p.q, by eight
// threads (j = 0..7 of `mask`): inverse_partition (:1173-1274) with its DC-only shortcut, a row or
// column each, the reconstruction SSE, and write_inter_scan's (:1414-1432) bits, eight scan slots
// each. tmp: 64 words of the eight threads' own.
__device__ void eval_octet(const TrdArgs& A, const TrdShared& sh, int j, unsigned mask, int k, int t, int mquant, int2 vis,
                           TParent& p, int* tmp) {
    const DevParams& P = A.P;
    const bool derived = A.cfg.dquantfrm != 0;  // the reference passes DQUANTFRM here
    const int np = part_count(t);
    auto dq = [&](int i) { return trd_dequant(P, p.q[i], mquant, derived); };
    uint32_t row = 0;
#pragma unroll
    for (int x = 0; x < 8; ++x) row |= p.q[j * 8 + x] ? 1u << x : 0u;
    const uint32_t lo = __reduce_or_sync(mask, j < 4 ? row << (8 * j) : 0u);
    const uint32_t hi = __reduce_or_sync(mask, j >= 4 ? row << (8 * (j - 4)) : 0u);
    const uint64_t cells = ((uint64_t)hi << 32) | lo;
    int s[8], o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = dq(t == 1 ? i * 8 + j : j * 8 + i);
    if (t <= 2) {
        inv8(s, 1, o, 1, 4, 3, 0);
    } else {
        inv4(s, 1, o, 1, 4, 3);
        inv4(s + 4, 1, o + 4, 1, 4, 3);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) tmp[j * 8 + i] = o[i];
    __syncwarp(mask);
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = tmp[i * 8 + j];
    if (t == 1 || t == 3) {
        inv8(s, 1, o, 1, 64, 7, 1);
    } else {
        inv4(s, 1, o, 1, 64, 7);
        inv4(s + 4, 1, o + 4, 1, 64, 7);
    }
    uint32_t sse = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // the column's upper and lower half lie in one partition each
        const int part = t == 1 ? 0 : (t == 2 ? h : (t == 3 ? j >> 2 : 2 * h + (j >> 2)));
        const int org = part_origin(t, part);
        const uint64_t own = cells & part_cells(t, part);
        const bool dc_only = own == (1ull << org);
        int dc = 0;
        if (dc_only) {
            dc = dq(org);
            dc = t <= 2 ? arshift(3 * dc + 1, 1) : arshift(17 * dc + 4, 3);
            dc = t == 1 ? arshift(3 * dc + 16, 5) : (t == 3 ? arshift(12 * dc + 64, 7) : arshift(17 * dc + 64, 7));
        }
#pragma unroll
        for (int i = 4 * h; i < 4 * h + 4; ++i) {
            const int r = dc_only ? dc : (own ? o[i] : 0);
            if (j < vis.x && i < vis.y) {
                const int e = (int)sh.src[k][i * 8 + j] - iclamp((int)sh.pred[k][i * 8 + j] + r, 0, 255);
                sse += (uint32_t)(e * e);
            }
        }
    }
    sse = __reduce_add_sync(mask, sse);
    // the coded coefficients in scan order: slot = partition * n + scan position
    int n;
    const uint8_t* scan = inter_scan(t, n);
    uint32_t slots = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int slot = 8 * j + i, part = slot / n;
        slots |= ((cells >> (part_origin(t, part) + scan[slot - part * n])) & 1) ? 1u << i : 0u;
    }
    const uint32_t slo = __reduce_or_sync(mask, j < 4 ? slots << (8 * j) : 0u);
    const uint32_t shi = __reduce_or_sync(mask, j >= 4 ? slots << (8 * (j - 4)) : 0u);
    const uint64_t coded = ((uint64_t)shi << 32) | slo;
    const int header = (P.pq < 8 || A.cfg.dquantfrm) ? 7 : 8;
    auto bits_of = [&](int slot) {
        const int part = slot / n;
        const uint64_t in = coded & ((n == 64 ? ~0ull : (1ull << n) - 1) << (part * n));
        const uint64_t before = in & ((1ull << slot) - 1);
        const int prev = before ? 63 - __clzll((long long)before) : part * n - 1;
        const bool last = (in >> slot) == 1;
        return ac_coeff_bits(A, slot - prev - 1, p.q[part_origin(t, part) + scan[slot - part * n]], last);
    };
    uint32_t none = 0, after = 0;  // no header written yet / already written
    int first = 64;                // the first coefficient that would write it
    for (uint32_t m = slots; m; m &= m - 1) {
        const int slot = 8 * j + __ffs(m) - 1;
        const CoeffBits b = bits_of(slot);
        if (b.other && b.other < b.esc3 + header) none += (uint32_t)b.other;
        else if (first == 64) first = slot;
        after += (uint32_t)((b.other && b.other < b.esc3) ? b.other : b.esc3);
    }
    first = __reduce_min_sync(mask, first);
    if (first < 64) {
        none = 0;
        for (uint32_t m = slots; m; m &= m - 1) {
            const int slot = 8 * j + __ffs(m) - 1;
            const CoeffBits b = bits_of(slot);
            none += (uint32_t)(slot < first ? b.other : slot == first ? b.esc3 + header
                                                      : ((b.other && b.other < b.esc3) ? b.other : b.esc3));
        }
    }
    none = __reduce_add_sync(mask, none);
    after = __reduce_add_sync(mask, after);
    if (j == 0) {
        int skip = 0;
        for (int part = 0; part < np; ++part)
            if (!(cells & part_cells(t, part))) skip |= 1 << (np - 1 - part);
        p.type = (uint8_t)t;
        p.skip = (uint8_t)skip;
        p.distortion = (double)sse;
        p.coef0 = none;
        p.coef1 = after;
        p.esc0 = first < 64;
        // estimate_parent_payload_bits (:1528-1543)
        uint32_t bits = 0;
        if (skip != (1 << np) - 1) {
            if (t == 4) bits += (uint32_t)subblkpat_bits(P, skip);
            else if (t == 2 || t == 3) bits += (uint32_t)rect_subblkpat_bits(skip);
            bits += none;
        }
        p.bits = bits;
    }
}

// An MbTransformDecision: parents by index into the parent pool
struct TDec {
    int8_t parent[6];
    uint8_t type, level, cbp;
    double distortion;
    uint32_t bits;
};

// refresh_transform_estimate (:1496-1526) with write_transform_payload (:1434-1494)
__device__ void refresh(const TrdArgs& A, TDec& d, const TParent* pool) {
    const DevParams& P = A.P;
    d.cbp = 0;
    d.distortion = 0.0;
    int first = -1;
    for (int k = 0; k < 6; ++k) {
        const TParent& p = pool[d.parent[k]];
        d.distortion += p.distortion;
        const int np = part_count(p.type);
        if (p.skip != (1 << np) - 1) {
            d.cbp |= (uint8_t)(1 << (5 - k));
            if (first < 0) first = k;
        }
    }
    if (first >= 0 && d.level == 1) d.type = pool[d.parent[first]].type;
    d.bits = 0;
    if (!d.cbp) return;
    uint32_t bits = ent::kPcbpBits[d.cbp];
    bool esc = false;
    const TParent& fp = pool[d.parent[first]];
    if (A.cfg.variable_transforms) {
        if (d.level == 0) bits += (uint32_t)ttmb_macro_bits(P, d.type, fp.skip);
        else if (d.level == 1) bits += (uint32_t)ttmb_block_bits(P, fp.type, fp.skip);
    }
    for (int k = 0; k < 6; ++k) {
        if (!(d.cbp & (1 << (5 - k)))) continue;
        const TParent& p = pool[d.parent[k]];
        const int t = p.type;
        if (A.cfg.variable_transforms) {
            if (d.level == 1) {
                if (k != first) bits += (uint32_t)ttblk_bits(P, t, p.skip);
                if (t == 4) bits += (uint32_t)subblkpat_bits(P, p.skip);
            } else if (d.level == 0) {
                if (t == 4) bits += (uint32_t)subblkpat_bits(P, p.skip);
                else if ((t == 2 || t == 3) && k != first) bits += (uint32_t)rect_subblkpat_bits(p.skip);
            } else {
                if (t == 4) bits += (uint32_t)subblkpat_bits(P, p.skip);
                else if (t == 2 || t == 3) bits += (uint32_t)rect_subblkpat_bits(p.skip);
            }
        }
        bits += esc ? p.coef1 : p.coef0;
        esc = esc || p.esc0;
    }
    d.bits = bits;
}

__device__ __forceinline__ double rd_of(const TDec& d, double lambda) { return d.distortion + lambda * (double)d.bits; }

// The trellis of every listed partition (jobs[i] = job * 4 + partition; the job's parent, type and
// coefficients by `job_of`), by teams of the block's threads.
template <int BEAM, class F>
__device__ __forceinline__ void trellis_jobs(const TrdArgs& A, TrdShared& sh, int mx, int my, int mquant, F job_of) {
    constexpr int G = TrellisMem<BEAM>::kTeam;
    const int tid = threadIdx.x, team = tid / G, lane = tid & 31;
    const Team g{G == 32 ? 0xffffffffu : 0xffffu << (lane & 16), tid % G, G};
    TrellisMem<BEAM>& mem = reinterpret_cast<TrellisMem<BEAM>*>(sh.trellis)[team];
    const DevParams& P = A.P;
    for (int i = team; i < sh.n_jobs; i += kTrdThreads / G) {
        const int job = sh.jobs[i] >> 2, part = sh.jobs[i] & 3;
        int k, t, cand, out;
        job_of(job, k, t, cand, out);
        int ox, oy, bw, bh;
        part_geometry(t, part, ox, oy, bw, bh);
        const bool chroma = k >= 4;
        const int x0 = (chroma ? mx : mx * 2 + (k & 1)) * 8 + ox, y0 = (chroma ? my : my * 2 + ((k >> 1) & 1)) * 8 + oy;
        const uint8_t* sp = chroma ? (k == 4 ? A.src.u : A.src.v) : A.src.y;
        const uint8_t* pp = chroma ? (k == 4 ? A.pred.u : A.pred.v) : A.pred.y;
        const int w = chroma ? P.W / 2 : P.W, h = chroma ? P.H / 2 : P.H;
        const int org = part_origin(t, part);
        double ls = 1.0;
        if (x0 < w && y0 < h)
            ls = aq_scale(g, A, sp, chroma ? A.src.pitch_c : A.src.pitch_y, w, h, x0, y0, bw, bh, pp,
                          chroma ? A.pred.pitch_c : A.pred.pitch_y, chroma ? A.src.y : nullptr, A.src.pitch_y);
        int n;
        const uint8_t* scan = inter_scan(t, n);
        trellis_team<BEAM>(g, A, sh.c[cand] + org, sh.sq[cand] + org, t, ls, mquant, scan, n, 0, false, sh.pool[out].q + org, mem);
    }
}

__global__ void __launch_bounds__(kTrdThreads) trd_kernel(const __grid_constant__ TrdArgs A) {
    __shared__ TrdShared sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int item = blockIdx.x;
    const DevParams& P = A.P;
    const int mb = A.mb_list ? A.mb_list[item] : item;
    const int mx = mb % P.mbw, my = mb / P.mbw;
    const int mquant = (A.mquant && A.mquant[mb] >= 1) ? (int)A.mquant[mb] : P.pq;
    const vc1cu_trd_cfg& cfg = A.cfg;
    // candidates whose decision is final at once: the 8x8-only and frame-level forms (with trellis)
    const bool direct = !cfg.variable_transforms || cfg.frame_type;
    const bool trellis = cfg.trellis > 0 && !(cfg.hrd_enabled && mquant == 1);  // else its levels are the scalar ones
    // ---- the macroblock's blocks ----
    for (int i = tid; i < 384; i += kTrdThreads) {
        const int k = i >> 6, x = i & 7, y = (i >> 3) & 7;
        const bool chroma = k >= 4;
        const int2 vis = block_extent(P, mx, my, k);
        const int gx = (chroma ? mx : mx * 2 + (k & 1)) * 8 + x, gy = (chroma ? my : my * 2 + ((k >> 1) & 1)) * 8 + y;
        int a = 0, b = 0;
        if (x < vis.x && y < vis.y) {
            a = __ldg((chroma ? (k == 4 ? A.src.u : A.src.v) : A.src.y) + (size_t)gy * (chroma ? A.src.pitch_c : A.src.pitch_y) + gx);
            b = __ldg((chroma ? (k == 4 ? A.pred.u : A.pred.v) : A.pred.y) + (size_t)gy * (chroma ? A.pred.pitch_c : A.pred.pitch_y) + gx);
        }
        sh.src[k][i & 63] = (uint8_t)a;
        sh.pred[k][i & 63] = (uint8_t)b;
        sh.px[k][i & 63] = (int16_t)(a - b);
    }
    __syncthreads();
    // ---- the candidate list, and beside it the macroblock's lambda scale ----
    if (warp == 0) {
        if (direct) {
            if (lane == 0) {
                sh.list[0] = cfg.variable_transforms ? cfg.frame_type : 1;
                sh.count = 1;
            }
        } else {
            // transform_metrics (transform_residual_metrics.h:29-61), each lane half a row
            const int py = lane >> 1, px0 = (lane & 1) * 8;
            uint32_t sad = 0, hedge = 0, vedge = 0, grad = 0;
            if (my * 16 + py < P.H) {
                auto R = [&](int x, int y) { return (int)sh.px[(y >> 3) * 2 + (x >> 3)][(y & 7) * 8 + (x & 7)]; };
                for (int px = px0; px < px0 + 8 && mx * 16 + px < P.W; ++px) {
                    const int r = R(px, py);
                    sad += (uint32_t)iabs(r);
                    if ((py & 7) == 4) hedge += (uint32_t)iabs(r - R(px, py - 1));
                    if ((px & 7) == 4) vedge += (uint32_t)iabs(r - R(px - 1, py));
                    if (px > 0) grad += (uint32_t)iabs(r - R(px - 1, py));
                    if (py > 0) grad += (uint32_t)iabs(r - R(px, py - 1));
                }
            }
            sad = __reduce_add_sync(0xffffffffu, sad);
            hedge = __reduce_add_sync(0xffffffffu, hedge);
            vedge = __reduce_add_sync(0xffffffffu, vedge);
            grad = __reduce_add_sync(0xffffffffu, grad);
            if (lane == 0) {
                const uint64_t S = sad, HE = hedge, VE = vedge, GR = grad, lim = (uint64_t)(64 * mquant);
                int l[4] = {1, 1, 1, 1}, count = 0;
                const bool split_x = mx == P.mbw - 1 && (P.W & 15) != 0, split_y = my == P.mbh - 1 && (P.H & 15) != 0;
                if (split_x && split_y) {
                    l[count++] = 4;
                } else if (split_x || split_y) {
                    l[count++] = split_x ? 3 : 2;
                    if (S > lim && GR > S * 2) l[count++] = 4;
                } else {
                    l[count++] = 1;
                    if (S > lim) {
                        if (HE * 5 > VE * 6) l[count++] = 2;
                        else if (VE * 5 > HE * 6) l[count++] = 3;
                        else { l[count++] = 2; l[count++] = 3; }
                        if (count < 4 && GR > S * 2) l[count++] = 4;
                    }
                }
                for (int i = 0; i < 4; ++i) sh.list[i] = l[i];
                sh.count = count;
            }
        }
    } else if (warp == 1 && !direct) {
        const Team g{0xffffffffu, lane, 32};
        const double ls = aq_scale(g, A, A.src.y, A.src.pitch_y, P.W, P.H, mx * 16, my * 16, 16, 16, A.pred.y, A.pred.pitch_y,
                                   nullptr, 0);
        if (lane == 0) sh.lscale = ls;
    }
    __syncthreads();
    const int count = sh.count, parents = 6 * count;
    // ---- every candidate's six parents: coefficients, scalar levels ----
    {
        int base = 0;
        for (int i = 0; i < count; ++i) {
            const int t = sh.list[i], per = xform_threads(t), bh = (t == 2 || t == 4) ? 4 : 8;
            // the first thread of a type follows the last of the one before it
            for (int task = (tid - base) & (kTrdThreads - 1); task < 6 * per; task += kTrdThreads) {
                const int k = task / per, sub = task - k * per;
                forward_row(sh.px[k], t, sub / bh, sub % bh, sh.c[i * 6 + k]);
            }
            base += 6 * per;
        }
    }
    __syncthreads();
    for (int i = tid; i < parents * 64; i += kTrdThreads) {
        const int v = trd_squant(P, sh.c[i >> 6][i & 63], mquant, mquant != P.pq);
        sh.sq[i >> 6][i & 63] = (int16_t)v;
        sh.pool[i >> 6].q[i & 63] = (int16_t)v;
    }
    if (tid == 0) {
        sh.n_jobs = 0;
        if (direct && trellis)
            for (int k = 0; k < 6; ++k)
                for (int part = 0; part < part_count(sh.list[0]); ++part) sh.jobs[sh.n_jobs++] = (uint8_t)(k * 4 + part);
    }
    __syncthreads();
    if (direct && trellis) {
        auto job_of = [&](int job, int& k, int& t, int& cand, int& out) {
            k = cand = out = job;
            t = sh.list[0];
        };
        if (cfg.trellis >= 2) trellis_jobs<8>(A, sh, mx, my, mquant, job_of);
        else trellis_jobs<4>(A, sh, mx, my, mquant, job_of);
        __syncthreads();
    }
    const int octet = tid >> 3, oj = tid & 7;
    const unsigned omask = 0xffu << (lane & 24);
    for (int i = octet; i < parents; i += kTrdThreads / 8)
        eval_octet(A, sh, oj, omask, i % 6, sh.list[i / 6], mquant, block_extent(P, mx, my, i % 6), sh.pool[i], sh.tmp[octet]);
    __syncthreads();
    // ---- the macroblock- and block-level winners ----
    TDec macro{}, block{};
    double lambda = 0.0;
    if (warp == 0) {
        if (direct) {
            if (lane == 0) {
                for (int k = 0; k < 6; ++k) macro.parent[k] = (int8_t)k;
                macro.type = (uint8_t)sh.list[0];
                macro.level = cfg.variable_transforms ? 2 : 0;
                refresh(A, macro, sh.pool);
            }
        } else {
            lambda = 0.75 * (double)(2 * mquant) * (double)(2 * mquant) * sh.lscale;
            // a candidate per lane; the first of the least
            TDec cand{};
            double rd = __longlong_as_double(0x7ff0000000000000LL);
            if (lane < count) {
                for (int k = 0; k < 6; ++k) cand.parent[k] = (int8_t)(lane * 6 + k);
                cand.type = (uint8_t)sh.list[lane];
                cand.level = 0;
                refresh(A, cand, sh.pool);
                rd = rd_of(cand, lambda);
            }
            int best_i = 0;
            double best_rd = __shfl_sync(0xffffffffu, rd, 0);
            for (int i = 1; i < count; ++i) {
                const double r = __shfl_sync(0xffffffffu, rd, i);
                if (r < best_rd) {
                    best_rd = r;
                    best_i = i;
                }
            }
            // a parent block per lane
            int bi = 0;
            if (lane < 6) {
                auto prd = [&](const TParent& p) {
                    return p.distortion + lambda * (double)(p.bits + parent_ttblk_bits(P, p));
                };
                double brd = prd(sh.pool[lane]);
                for (int i = 1; i < count; ++i) {
                    const double r = prd(sh.pool[i * 6 + lane]);
                    if (r < brd) {
                        brd = r;
                        bi = i;
                    }
                }
            }
            for (int k = 0; k < 6; ++k) block.parent[k] = (int8_t)(__shfl_sync(0xffffffffu, bi, k) * 6 + k);
            // the winner's estimate from its lane, the block decision's on lane 0
            macro.distortion = __shfl_sync(0xffffffffu, cand.distortion, best_i);
            macro.bits = __shfl_sync(0xffffffffu, cand.bits, best_i);
            macro.cbp = (uint8_t)__shfl_sync(0xffffffffu, (int)cand.cbp, best_i);
            macro.type = (uint8_t)__shfl_sync(0xffffffffu, (int)cand.type, best_i);
            if (lane == 0) {
                for (int k = 0; k < 6; ++k) macro.parent[k] = (int8_t)(best_i * 6 + k);
                macro.level = 0;
                block.type = (uint8_t)sh.list[0];
                block.level = 1;
                refresh(A, block, sh.pool);
                sh.macro_type = macro.type;
                int n = 0;
                for (int job = 0; job < 12; ++job) {
                    const int k = job % 6, t = job < 6 ? macro.type : sh.pool[block.parent[k]].type;
                    if (job >= 6) sh.need[k] = (uint8_t)t;
                    if (job >= 6 && t == macro.type) continue;
                    for (int part = 0; part < part_count(t); ++part) sh.jobs[n++] = (uint8_t)(job * 4 + part);
                }
                sh.n_jobs = n;
            }
        }
    }
    // ---- trellis re-evaluation of the macroblock winner and of the block winners of other types ----
    if (!direct && cfg.trellis > 0) {
        __syncthreads();
        auto job_of = [&](int job, int& k, int& t, int& cand, int& out) {
            k = job % 6;
            t = job < 6 ? sh.macro_type : sh.need[k];
            int i = 0;
            while (i < 3 && sh.list[i] != t) ++i;
            cand = i * 6 + k;
            out = 24 + job;
        };
        if (!trellis) {
            for (int i = tid; i < 12 * 64; i += kTrdThreads) {
                int k, t, cand, out;
                job_of(i >> 6, k, t, cand, out);
                sh.pool[out].q[i & 63] = sh.sq[cand][i & 63];
            }
        } else if (cfg.trellis >= 2) {
            trellis_jobs<8>(A, sh, mx, my, mquant, job_of);
        } else {
            trellis_jobs<4>(A, sh, mx, my, mquant, job_of);
        }
        __syncthreads();
        if (octet < 12) {
            int k, t, cand, out;
            job_of(octet, k, t, cand, out);
            if (octet < 6 || t != sh.macro_type)
                eval_octet(A, sh, oj, omask, k, t, mquant, block_extent(P, mx, my, k), sh.pool[out], sh.tmp[octet]);
        }
        __syncthreads();
        if (tid == 0) {
            for (int k = 0; k < 6; ++k) macro.parent[k] = (int8_t)(24 + k);
            macro.level = 0;
            refresh(A, macro, sh.pool);
            for (int k = 0; k < 6; ++k) block.parent[k] = (int8_t)(sh.need[k] == sh.macro_type ? 24 + k : 30 + k);
            block.level = 1;
            refresh(A, block, sh.pool);
        }
    }
    // ---- the signaling decision and the outputs ----
    if (tid == 0) {
        TDec d = macro;
        if (!direct && cfg.extended_transform_signaling && rd_of(block, lambda) < rd_of(macro, lambda) * 0.9999) d = block;
        vc1cu_tdecision o{};
        o.type = d.type;
        o.signal_level = d.level;
        o.cbp = d.cbp;
        o.estimated_bits = d.bits;
        o.distortion = d.distortion;
        for (int k = 0; k < 6; ++k) {
            const TParent& p = sh.pool[d.parent[k]];
            o.parent_type[k] = p.type;
            o.skip_mask[k] = p.skip;
            o.parent_bits[k] = p.bits;
            o.parent_distortion[k] = p.distortion;
            sh.chosen[k] = d.parent[k];
        }
        A.out[item] = o;
    }
    __syncthreads();
    if (A.levels)
        for (int i = tid; i < 6 * 64; i += kTrdThreads) A.levels[(size_t)item * 384 + i] = sh.pool[sh.chosen[i >> 6]].q[i & 63];
}

// ---- I-picture intra reconstruction (reconstruct_i_signed_padded, encoder_encode.cpp:814-887) ----

// dc_scale (encoder_entropy.cpp:369-375): the DC step of MQUANT 1..31
__device__ __forceinline__ int intra_dc_scale(int q) {
    return q <= 0 ? 0 : (q == 1 ? 2 : (q == 2 ? 4 : (q <= 5 ? 8 : q / 2 + 6)));
}
// DQScale (SMPTE 421M 8.1.3.4, dqscale_value :434-447): round(2^18 / n) for n = index + 1
__device__ __forceinline__ int intra_dqscale(int index) {
    const int n = index + 1;
    return (0x40000 + n / 2) / n;
}
// reconstruct_dc_sample_with_bias (:383-389)
__device__ __forceinline__ int intra_dc_sample(int qdc, int mq, int bias) {
    int x = qdc * intra_dc_scale(mq);
    x = arshift(3 * x + 1, 1);
    x = arshift(3 * x + 16, 5);
    return min(255, max(0, bias + x));
}
// choose_dc_for_mean_with_bias (:395-412): the DC level whose reconstruction is nearest the mean
__device__ int intra_dc_for_mean(int mean, int mq, int bias) {
    const int bits = 8 + ((mq == 1 || mq == 2) ? 3 - mq : 0);
    const int maxq = (1 << bits) - 1;
    int lo = -maxq, hi = maxq;
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2;
        if (intra_dc_sample(mid, mq, bias) < mean) lo = mid + 1;
        else hi = mid;
    }
    int best = lo;
    if (lo > -maxq && iabs(intra_dc_sample(lo - 1, mq, bias) - mean) <= iabs(intra_dc_sample(lo, mq, bias) - mean)) best = lo - 1;
    return best;
}
// scale_dc_predictor (:449-456)
__device__ __forceinline__ int intra_scale_dc(int value, int from_q, int to_q) {
    from_q = iabs(from_q);
    to_q = iabs(to_q);
    if (!from_q || from_q == to_q) return value;
    const int idx = intra_dc_scale(to_q) - 1;
    if (idx < 0) return 0;
    const long long v = (long long)value * intra_dc_scale(from_q) * intra_dqscale(idx);
    return (int)((v + 0x20000) >> 18);
}

// The intra source, its MQUANT map and the per-block outputs of one I picture.
struct IntraArgs {
    DevParams P;
    const uint8_t* y;
    const uint8_t* u;
    const uint8_t* v;
    int pitch_y, pitch_c, sw, sh;  // the intra source's luma raster (the picture or its edge source)
    const uint8_t* mquant;         // per MB (nullptr: PQINDEX)
    const uint8_t* derived;        // per MB DQUANT-derived flag (nullptr: none)
    int16_t* q;                    // [mb][6][64] AC levels
    int* dc[3];                    // per plane block grid: the DC target, then the final DC
    int* qg[3];                    // per plane block grid: MQUANT, negative when derived
    TrdArgs trd;                   // P, tab, cfg (trellis, hrd_enabled, AQ) and the intra source's luma mean
};

__device__ __forceinline__ int intra_mq(const IntraArgs& A, int mb) {
    return (A.mquant && A.mquant[mb] >= 1) ? (int)A.mquant[mb] : A.P.pq;
}

// One block of threads per MB: forward_transform (:672-795; samples outside the source read the
// pad value, 0 luma / 128 chroma, minus 128), the AC levels of quantize_ac (:2090-2144: scalar, or
// the trellis along the intra scan from position 1 with the intra-family rates and the perceptual
// lambda scale of the block, chroma weighed against the intra source's luma) and
// choose_dc_for_mean of the padded block mean. The stages are the transform RD's: one transform row
// and one coefficient per thread, sixteen (32) threads per trellis. One thread per block took 0.5 ms
// per 720p picture with the trellis.
__global__ void __launch_bounds__(kTrdThreads) intra_fwd_kernel(const __grid_constant__ IntraArgs A) {
    __shared__ double c[6][64];
    __shared__ int16_t px[6][64], sq[6][64], lv[6][64];
    __shared__ unsigned sums[6];
    __shared__ alignas(16) uint8_t trellis_mem[kTrellisBytes + 1024];
    const DevParams& P = A.P;
    const int tid = threadIdx.x, lane = tid & 31, mb = blockIdx.x, mx = mb % P.mbw, my = mb / P.mbw;
    const int mq = intra_mq(A, mb);
    const bool trellis = A.trd.cfg.trellis > 0 && !(A.trd.cfg.hrd_enabled && mq == 1);
    // the scalar levels the trellis starts from take its own rule for the half step
    const bool derived = trellis ? mq != P.pq : (A.derived && A.derived[mb]);
    if (tid < 6) sums[tid] = 0;
    __syncthreads();
    for (int i = tid; i < 384; i += kTrdThreads) {
        const int k = i >> 6;
        const bool chroma = k >= 4;
        const uint8_t* p = chroma ? (k == 4 ? A.u : A.v) : A.y;
        const int pitch = chroma ? A.pitch_c : A.pitch_y, w = chroma ? A.sw / 2 : A.sw, h = chroma ? A.sh / 2 : A.sh;
        const int sx = (chroma ? mx : mx * 2 + (k & 1)) * 8 + (i & 7), sy = (chroma ? my : my * 2 + ((k >> 1) & 1)) * 8 + ((i >> 3) & 7);
        const int v = (sx < w && sy < h) ? (int)__ldg(p + (size_t)sy * pitch + sx) : (chroma ? 128 : 0);
        px[k][i & 63] = (int16_t)(v - 128);
        const unsigned s = __reduce_add_sync(0xffffffffu, (unsigned)v);  // a warp's 32 samples lie in one block
        if (lane == 0) atomicAdd(&sums[k], s);
    }
    __syncthreads();
    if (tid < 48) forward_row(px[tid >> 3], 1, 0, tid & 7, c[tid >> 3]);
    __syncthreads();
    for (int i = tid; i < 384; i += kTrdThreads) {
        const int k = i >> 6, j = i & 63;
        const int v = j ? trd_squant(P, c[k][j], mq, derived) : 0;
        if (!j) c[k][0] = 0.0;  // the DC stays out of the trellis (first_scan 1)
        sq[k][j] = (int16_t)v;
        lv[k][j] = (int16_t)v;
    }
    __syncthreads();
    if (trellis) {
        auto block = [&](const Team& g, int k, auto& mem, auto run) {
            const bool chroma = k >= 4;
            const uint8_t* p = chroma ? (k == 4 ? A.u : A.v) : A.y;
            const int x0 = (chroma ? mx : mx * 2 + (k & 1)) * 8, y0 = (chroma ? my : my * 2 + ((k >> 1) & 1)) * 8;
            // the luma context is read as a coded-width raster (stats(*luma_context, width, height, ...)):
            // an edge source of a cropped picture is a padded-width raster read at the coded width
            const int lpitch = A.sw == P.W ? A.pitch_y : P.W;
            const double ls = aq_scale(g, A.trd, p, chroma ? A.pitch_c : A.pitch_y, chroma ? A.sw / 2 : A.sw,
                                       chroma ? A.sh / 2 : A.sh, x0, y0, 8, 8, nullptr, 0, chroma ? A.y : nullptr, lpitch);
            run(g, k, ls, !chroma, mem);
        };
        if (A.trd.cfg.trellis >= 2) {
            TrellisMem<8>& mem = reinterpret_cast<TrellisMem<8>*>(trellis_mem)[tid / 32];
            for (int k = tid / 32; k < 6; k += kTrdThreads / 32)
                block(Team{0xffffffffu, lane, 32}, k, mem, [&](const Team& g, int kk, double ls, bool intra, TrellisMem<8>& m) {
                    trellis_team<8>(g, A.trd, c[kk], sq[kk], 1, ls, mq, ent::kIntraScan, 64, 1, intra, lv[kk], m);
                });
        } else {
            TrellisMem<4>& mem = reinterpret_cast<TrellisMem<4>*>(trellis_mem)[tid / 16];
            const int k = tid / 16;
            if (k < 6)
                block(Team{0xffffu << (lane & 16), tid & 15, 16}, k, mem,
                      [&](const Team& g, int kk, double ls, bool intra, TrellisMem<4>& m) {
                          trellis_team<4>(g, A.trd, c[kk], sq[kk], 1, ls, mq, ent::kIntraScan, 64, 1, intra, lv[kk], m);
                      });
        }
        __syncthreads();
    }
    for (int i = tid; i < 384; i += kTrdThreads) A.q[(size_t)mb * 384 + i] = lv[i >> 6][i & 63];
    if (tid < 6) {
        const bool chroma = tid >= 4;
        const int bx = chroma ? mx : mx * 2 + (tid & 1), by = chroma ? my : my * 2 + ((tid >> 1) & 1);
        const int gw = chroma ? P.mbw : P.mbw * 2;
        A.dc[chroma ? tid - 3 : 0][by * gw + bx] = intra_dc_for_mean((int)((sums[tid] + 32u) / 64u), mq, 128);
    }
}

// predict_dc_dquant + clamp_dc_target_for_diff (encoder_entropy.cpp:549-571, :426-432) along the
// block grid of plane blockIdx.x (0 luma, 1 U, 2 V): a block's prediction reads its left, top
// and top-left neighbours' final DC, so the grid is walked by anti-diagonals.
__global__ void intra_dc_kernel(const __grid_constant__ IntraArgs A) {
    const DevParams& P = A.P;
    const int pl = blockIdx.x;
    const int gw = pl ? P.mbw : P.mbw * 2, gh = pl ? P.mbh : P.mbh * 2;
    int* g = A.dc[pl];
    int* qg = A.qg[pl];
    for (int d = 0; d < gw + gh - 1; ++d) {
        for (int y = max(0, d - gw + 1) + (int)threadIdx.x; y <= min(d, gh - 1); y += blockDim.x) {
            const int x = d - y;
            const int mb = pl ? y * P.mbw + x : (y >> 1) * P.mbw + (x >> 1);
            const int mq = intra_mq(A, mb);
            const bool a_avail = y > 0, c_avail = x > 0;
            int a = 0, b = 0, c = 0;
            if (a_avail) a = intra_scale_dc(g[(y - 1) * gw + x], qg[(y - 1) * gw + x], mq);
            if (c_avail) c = intra_scale_dc(g[y * gw + x - 1], qg[y * gw + x - 1], mq);
            if (a_avail && c_avail) b = intra_scale_dc(g[(y - 1) * gw + x - 1], qg[(y - 1) * gw + x - 1], mq);
            const bool left = c_avail && (!a_avail || iabs(a - b) <= iabs(b - c));
            const int pred = left ? c : (a_avail ? a : 0);
            const int bits = 8 + ((mq == 1 || mq == 2) ? 3 - mq : 0);
            const int maxv = (1 << bits) - 1;
            const int diff = min(maxv, max(-maxv, g[y * gw + x] - pred));
            g[y * gw + x] = min(maxv, max(-maxv, pred + diff));
            qg[y * gw + x] = (A.derived && A.derived[mb]) ? -mq : mq;
        }
        __syncthreads();
    }
}

// One thread per (MB, block): the coefficients (DC * dc_scale, dequant_level of the AC levels),
// inverse_transform_8x8 and the signed samples into the padded raster (rows packed).
__global__ void intra_inv_kernel(const __grid_constant__ IntraArgs A, int32_t* oy, int32_t* ou, int32_t* ov) {
    const DevParams& P = A.P;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.mbw * P.mbh * 6) return;
    const int mb = i / 6, k = i % 6, mx = mb % P.mbw, my = mb / P.mbw;
    const bool chroma = k >= 4;
    const int bx = chroma ? mx : mx * 2 + (k & 1), by = chroma ? my : my * 2 + ((k >> 1) & 1);
    const int gw = chroma ? P.mbw : P.mbw * 2;
    const int mq = intra_mq(A, mb);
    const bool derived = A.derived && A.derived[mb];
    const int16_t* q = A.q + (size_t)i * 64;
    int a[64], tmp[64];
    a[0] = A.dc[chroma ? k - 3 : 0][by * gw + bx] * intra_dc_scale(mq);
    for (int j = 1; j < 64; ++j) a[j] = trd_dequant(P, q[j], mq, derived);
    for (int j = 0; j < 64; ++j) tmp[j] = 0;
    for (int col = 0; col < 8; ++col) inv8(a + col, 8, tmp + col * 8, 1, 4, 3, 0);
    for (int col = 0; col < 8; ++col) inv8(tmp + col, 8, a + col, 8, 64, 7, 1);
    int32_t* o = chroma ? (k == 4 ? ou : ov) : oy;
    const int ow = chroma ? P.mbw * 8 : P.mbw * 16;
    for (int y = 0; y < 8; ++y)
        for (int x = 0; x < 8; ++x) o[(size_t)(by * 8 + y) * ow + bx * 8 + x] = a[y * 8 + x];
}

// make_overlap_edge_source (encoder_encode.cpp:13-63): the picture on the coded (whole-MB)
// raster with the samples beyond the visible crop replaced by the nearest visible sample along an
// active overlap edge (all edges, or those between two flagged macroblocks). One thread per
// destination sample of one plane (blockIdx.y).
__host__ __device__ inline int ovl_border(int visible, int coded) {
    if (visible < 1 || visible >= coded) return -1;
    const int rem = visible & 7;
    const int edge = rem == 7 ? visible + 1 : (rem == 0 ? visible : (rem == 1 ? visible - 1 : -1));
    return edge > 0 && edge < coded ? edge : -1;
}

struct EdgeArgs {
    const uint8_t* in[3];
    int in_pitch[3], sw[3], sh[3];
    uint8_t* out[3];
    int out_pitch[3], dw[3], dh[3], vw[3], vh[3], ex[3], ey[3];
    const uint8_t* flags;
    int all, mbw, mbh;
};

__global__ void edge_source_kernel(const __grid_constant__ EdgeArgs E) {
    const int pl = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= E.dw[pl] * E.dh[pl]) return;
    const int x = i % E.dw[pl], y = i / E.dw[pl];
    const bool luma = pl == 0;
    const int vw = E.vw[pl], vh = E.vh[pl];
    int v = (x < E.sw[pl] && y < E.sh[pl]) ? (int)E.in[pl][(size_t)y * E.in_pitch[pl] + x] : (luma ? 0 : 128);
    if (!(x < vw && y < vh)) {
        auto active = [&](int ax, int ay, int bx2, int by2) {
            if (E.all) return true;
            const int a = (luma ? ay / 2 : ay) * E.mbw + (luma ? ax / 2 : ax);
            const int b = (luma ? by2 / 2 : by2) * E.mbw + (luma ? bx2 / 2 : bx2);
            const int n = E.mbw * E.mbh;
            return a >= 0 && b >= 0 && a < n && b < n && E.flags[a] && E.flags[b];
        };
        const int ex = E.ex[pl], ey = E.ey[pl];
        const bool right = x >= vw && ex >= 0 && active(ex / 8 - 1, y / 8, ex / 8, y / 8);
        const bool bottom = y >= vh && ey >= 0 && active(x / 8, ey / 8 - 1, x / 8, ey / 8);
        if (right || bottom) {
            const int sx = min(max(x, 0), vw - 1), sy = min(max(y, 0), vh - 1);
            v = E.in[pl][(size_t)sy * E.in_pitch[pl] + sx];
        }
    }
    E.out[pl][(size_t)y * E.out_pitch[pl] + x] = (uint8_t)v;
}

// The DQUANT search's per-macroblock inputs (choose_dquant_transform_mb, encoder_aq.cpp:318-336):
// the perceptual lambda scale of the MB's luma against its prediction with its adjacency term,
// and the bright-detail-on-dark test of the source MB. One warp per MB.
__global__ void __launch_bounds__(128) dquant_stats_kernel(const __grid_constant__ TrdArgs A, double* lscale,
                                                           double* adjacency, uint8_t* bright) {
    const DevParams& P = A.P;
    const int mb = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (mb >= P.mbw * P.mbh) return;
    const Team g{0xffffffffu, (int)(threadIdx.x & 31), 32};
    const int x0 = (mb % P.mbw) * 16, y0 = (mb / P.mbw) * 16;
    double adj = 0.0;
    const double ls = aq_scale(g, A, A.src.y, A.src.pitch_y, P.W, P.H, x0, y0, 16, 16, A.pred.y, A.pred.pitch_y, nullptr, 0, &adj);
    uint32_t sum = 0, n = 0, hi = 0, lo = 0;
    for (int i = g.lane; i < 256; i += 32) {
        const int x = x0 + (i & 15), y = y0 + (i >> 4);
        if (x >= P.W || y >= P.H) continue;
        const int v = A.src.y[(size_t)y * A.src.pitch_y + x];
        sum += (uint32_t)v;
        ++n;
        hi += v >= 180;
        lo += v <= 48;
    }
    sum = g.sum(sum);
    n = g.sum(n);
    hi = g.sum(hi);
    lo = g.sum(lo);
    if (g.lane == 0) {
        lscale[mb] = ls;
        adjacency[mb] = adj;
        const double mean = n ? (double)sum / (int)n : 128.0;
        bright[mb] = (n && mean < 90.0 && (int)hi >= imax(2, (int)n / 32) && lo >= n / 2) ? 1 : 0;
    }
}

// mean of the source luma plane (cached_luma_mean, encoder_aq.cpp:506-545): one block's partial sums
__global__ void luma_sum_kernel(const uint8_t* y, int pitch, int W, int H, unsigned long long* sum) {
    unsigned long long s = 0;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < (long)W * H; i += (long)gridDim.x * blockDim.x)
        s += y[(size_t)(i / W) * pitch + i % W];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(sum, s);
}

}  // namespace

// The escape lengths on the host (ent::kAcEscapeBits lives in constant memory here).
static int ent_escape_bits(int set) {
    constexpr uint8_t bits[8] = {9, 9, 7, 9, 7, 7, 7, 7};
    return bits[set];
}

// The dense rate tables from the code lengths (host side).
size_t trd_tables_bytes() { return sizeof(TrdTables); }
void trd_fill_tables(void* host) {
    TrdTables& t = *static_cast<TrdTables*>(host);
    std::memset(&t, 0, sizeof t);
    std::memset(t.max_run, -1, sizeof t.max_run);
    for (int i = 0; i < ent::kAcEntries; ++i) {
        const uint8_t* e = ent::kAcEntry[i];
        const int set = e[0], run = e[1], level = e[2], last = e[3], bits = e[4];
        t.ac_bits[set][last][run][level] = (uint8_t)bits;
        if (level > t.max_level[set][last][run]) t.max_level[set][last][run] = (uint8_t)level;
        if (run > t.max_run[set][last][level]) t.max_run[set][last][level] = (int8_t)run;
    }
    // trellis_rate_bits_for_set (encoder_transform.cpp:1811-1841)
    auto direct = [&](int set, int run, int level, int last) {
        return run < 0 || run > 63 || level < 0 || level > 63 ? 0 : (int)t.ac_bits[set][last][run][level];
    };
    auto rate = [&](int run, int mag, int last, int set, int level_bits) {
        if (const int d = direct(set, run, mag, last)) return d + 1;
        const int esc = ent_escape_bits(set);
        int best = 1000000;
        const int level_delta = t.max_level[set][last][run];
        if (set != 3 && level_delta > 0 && mag > level_delta)
            if (const int b = direct(set, run, mag - level_delta, last)) best = esc + 1 + b + 1;
        const int run_delta = mag < 64 ? t.max_run[set][last][mag] : -1;
        if (run_delta >= 0 && run > run_delta)
            if (const int b = direct(set, run - run_delta - 1, mag, last)) best = std::min(best, esc + 2 + b + 1);
        return std::min(best, esc + 2 + 1 + 6 + 1 + level_bits);
    };
    // trellis_rate_bits (:1843-1857): the lower envelope of coding sets 1, 3, 5 (inter family) or 0, 2, 4
    // (intra family)
    for (int intra = 0; intra < 2; ++intra)
        for (int fine = 0; fine < 2; ++fine)
            for (int last = 0; last < 2; ++last)
                for (int run = 0; run < 64; ++run)
                    for (int mag = 1; mag < 128; ++mag) {
                        int bits = 1000000;
                        for (int set = intra ? 0 : 1; set <= 5; set += 2)
                            bits = std::min(bits, rate(run, mag, last, set, fine ? 11 : 8));
                        t.family[intra][fine][last][run][mag] = (uint8_t)bits;
                    }
}

// The source luma mean the perceptual lambda scale reads (0 when the scale is off).
static cudaError_t frame_mean_for(const DevParams& P, const DevFrame& src, const vc1cu_trd_cfg& cfg,
                                  unsigned long long* d_sum, cudaStream_t s, double& mean) {
    mean = 0.0;
    if (!cfg.adaptive_quality || cfg.aq_strength <= 0.0 || P.W <= 0 || P.H <= 0) return cudaSuccess;
    cudaError_t e;
    unsigned long long sum = 0;
    if ((e = cudaMemsetAsync(d_sum, 0, sizeof(unsigned long long), s)) != cudaSuccess) return e;
    luma_sum_kernel<<<148, 256, 0, s>>>(src.y, src.pitch_y, P.W, P.H, d_sum);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(&sum, d_sum, sizeof sum, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    mean = (double)sum / (double)((size_t)P.W * P.H);
    return cudaSuccess;
}

cudaError_t launch_trd(const DevParams& P, const DevFrame& src, const DevFrame& pred, const void* tables,
                       const uint8_t* mquant, const vc1cu_trd_cfg& cfg, unsigned long long* d_sum, vc1cu_tdecision* out,
                       int16_t* levels, cudaStream_t s, const int* mb_list, int n_list, double frame_mean) {
    cudaError_t e;
    if (frame_mean < 0.0 && (e = frame_mean_for(P, src, cfg, d_sum, s, frame_mean)) != cudaSuccess) return e;
    TrdArgs a;
    a.P = P;
    a.src = src;
    a.pred = pred;
    a.tab = static_cast<const TrdTables*>(tables);
    a.mquant = mquant;
    a.cfg = cfg;
    a.frame_mean = frame_mean < 0.0 ? 0.0 : frame_mean;
    a.out = out;
    a.levels = levels;
    a.mb_list = mb_list;
    a.n_list = n_list;
    const int items = mb_list ? n_list : P.mbw * P.mbh;
    if (items <= 0) return cudaSuccess;
    trd_kernel<<<items, kTrdThreads, 0, s>>>(a);
    return cudaGetLastError();
}

// The source luma mean of the perceptual lambda scale (for launches that share it).
cudaError_t trd_frame_mean(const DevParams& P, const DevFrame& src, const vc1cu_trd_cfg& cfg, unsigned long long* d_sum,
                           cudaStream_t s, double* mean) {
    return frame_mean_for(P, src, cfg, d_sum, s, *mean);
}

// The DQUANT search's per-MB scale, adjacency and bright-on-dark flags.
cudaError_t launch_dquant_stats(const DevParams& P, const DevFrame& src, const DevFrame& pred, const vc1cu_trd_cfg& cfg,
                                double frame_mean, double* lscale, double* adjacency, uint8_t* bright, cudaStream_t s) {
    TrdArgs a{};
    a.P = P;
    a.src = src;
    a.pred = pred;
    a.cfg = cfg;
    a.frame_mean = frame_mean;
    const int mbs = P.mbw * P.mbh;
    if (mbs <= 0) return cudaSuccess;
    dquant_stats_kernel<<<(mbs + 3) / 4, 128, 0, s>>>(a, lscale, adjacency, bright);
    return cudaGetLastError();
}

// The signed intra reconstruction of an I picture: the optional overlap edge source (flags: per
// MB, nullptr with all = 0 for none), the forward transforms and AC levels, the DC chain, the
// inverse transforms into the int32 planes oy / ou / ov (padded raster, rows packed). scratch
// holds intra_scratch_bytes(P) bytes; edge: 1.5 * (mbw * 16) * (mbh * 16) bytes for the edge
// source. tables / cfg: the AC length tables and the trellis and perceptual settings (trellis 0:
// scalar levels); the trellis's lambda scale reads the intra source's luma mean, taken here.
size_t intra_scratch_bytes(const DevParams& P) {
    const size_t mbs = (size_t)P.mbw * P.mbh;
    return mbs * 6 * 64 * 2 + mbs * 6 * 4 * 2 + 256;
}

cudaError_t launch_intra_recon(const DevParams& P, const DevFrame& src, int overlap, const uint8_t* d_flags,
                               const uint8_t* d_mquant, const uint8_t* d_derived, void* scratch, uint8_t* edge,
                               int32_t* oy, int32_t* ou, int32_t* ov, const void* tables, const vc1cu_trd_cfg& cfg,
                               cudaStream_t s) {
    const int mbs = P.mbw * P.mbh;
    if (mbs <= 0) return cudaSuccess;
    IntraArgs A{};
    A.P = P;
    A.y = src.y;
    A.u = src.u;
    A.v = src.v;
    A.pitch_y = src.pitch_y;
    A.pitch_c = src.pitch_c;
    A.sw = P.W;
    A.sh = P.H;
    cudaError_t e;
    if (overlap) {
        const int cw = P.mbw * 16, ch = P.mbh * 16, ccw = cw / 2, cch = ch / 2;
        const int cvw = (P.vw + 1) / 2, cvh = (P.vh + 1) / 2;
        const int vx = ovl_border(P.vw, cw), vy = ovl_border(P.vh, ch), cx = ovl_border(cvw, ccw), cy = ovl_border(cvh, cch);
        if (vx >= 0 || vy >= 0 || cx >= 0 || cy >= 0) {
            EdgeArgs E{};
            const uint8_t* in[3] = {src.y, src.u, src.v};
            for (int k = 0; k < 3; ++k) {
                const bool l = k == 0;
                E.in[k] = in[k];
                E.in_pitch[k] = l ? src.pitch_y : src.pitch_c;
                E.sw[k] = l ? P.W : P.W / 2;
                E.sh[k] = l ? P.H : P.H / 2;
                E.dw[k] = l ? cw : ccw;
                E.dh[k] = l ? ch : cch;
                E.out_pitch[k] = E.dw[k];
                E.vw[k] = l ? P.vw : cvw;
                E.vh[k] = l ? P.vh : cvh;
                E.ex[k] = l ? vx : cx;
                E.ey[k] = l ? vy : cy;
            }
            E.out[0] = edge;
            E.out[1] = edge + (size_t)cw * ch;
            E.out[2] = edge + (size_t)cw * ch + (size_t)ccw * cch;
            E.flags = d_flags;
            E.all = overlap == 1;
            E.mbw = P.mbw;
            E.mbh = P.mbh;
            edge_source_kernel<<<dim3((unsigned)((cw * ch + 255) / 256), 3), 256, 0, s>>>(E);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            A.y = E.out[0];
            A.u = E.out[1];
            A.v = E.out[2];
            A.pitch_y = cw;
            A.pitch_c = ccw;
            A.sw = cw;
            A.sh = ch;
        }
    }
    A.mquant = d_mquant;
    A.derived = d_derived;
    uint8_t* p = static_cast<uint8_t*>(scratch);
    A.q = reinterpret_cast<int16_t*>(p);
    p += (size_t)mbs * 6 * 64 * 2;
    int* dc = reinterpret_cast<int*>(p);
    int* qg = dc + (size_t)mbs * 6;
    A.dc[0] = dc;
    A.dc[1] = dc + (size_t)mbs * 4;
    A.dc[2] = dc + (size_t)mbs * 5;
    A.qg[0] = qg;
    A.qg[1] = qg + (size_t)mbs * 4;
    A.qg[2] = qg + (size_t)mbs * 5;
    A.trd.P = P;
    A.trd.tab = static_cast<const TrdTables*>(tables);
    A.trd.cfg = cfg;
    A.trd.frame_mean = 0.0;
    if (cfg.trellis > 0) {  // cached_luma_mean of the intra source's luma (the picture or its edge source)
        DevParams sp = P;
        sp.W = A.sw;
        sp.H = A.sh;
        DevFrame sf{};
        sf.y = A.y;
        sf.pitch_y = A.pitch_y;
        unsigned long long* d_sum = reinterpret_cast<unsigned long long*>(qg + (size_t)mbs * 6);
        if ((e = frame_mean_for(sp, sf, cfg, d_sum, s, A.trd.frame_mean)) != cudaSuccess) return e;
    }
    const unsigned blocks = (unsigned)((mbs * 6 + 127) / 128);
    intra_fwd_kernel<<<(unsigned)mbs, kTrdThreads, 0, s>>>(A);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    intra_dc_kernel<<<3, 256, 0, s>>>(A);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    intra_inv_kernel<<<blocks, 128, 0, s>>>(A, oy, ou, ov);
    return cudaGetLastError();
}

}  // namespace vc1cu
