// k_pipe.cu -- fused per-view pipeline kernels.
//
// Every fused kernel keeps the reference's per-entry arithmetic (the same
// operands combined in the same order with round-to-nearest float ops), so the
// fused pipeline is bit-identical to the composed module kernels and to the
// reference; fusion only removes HBM round trips and adds on-chip reuse.
//
//   k_prep_records  per pixel one 16-byte record: 64-bit census code, packed RGB
//   k_cost_volume   AD / census / AD+census(CombineCost) cost volume from records
//   (the cross-based stages work over view tables and live in k_batch.cu)
//   k_aw_wta        adaptive-weight aggregation (seq/AdaptiveWeightAggregation.cpp:73-111)
//                   over 64-pixel x 64-disparity tiles, weights made on the fly from
//                   Lab + host tables, and the arg-min over d
#include <algorithm>

#include "rts_fused.cuh"
#include "rts_pipe.h"
#include "rts_tma.h"
#include "rts_views.h"

namespace rts {

// ---------------------------------------------------------------------------
// Block per 64 x 16 pixels, the gray census window around them (wrapped,
// seq/CensusTransform.cpp:20-26) staged in shared memory, a thread on four pixels.  WIN: the
// 9x7 window, its 63 comparisons unrolled (a subtraction and a funnel shift of its sign
// bit each; the order of a code's bits is the same in all records of a launch and only
// distances of codes are used).  Bound: instruction issue.  1920x1080: 120 us an image
// with the window as loops over the image itself.
constexpr int kRecTW = 64, kRecTH = 16, kRecT = 256;
template <bool WIN>
__global__ void __launch_bounds__(kRecT) k_prep_records(const uint8_t *__restrict__ gray,
                                                        const uint8_t *__restrict__ rgb, uint4 *__restrict__ rec, int H,
                                                        int W, int hr_, int wr_, int want_code) {
    extern __shared__ uint8_t gt[];  // [16 + 2 hr][64 + 2 wr]
    const int hr = WIN ? 4 : hr_, wr = WIN ? 3 : wr_;
    const int gw = kRecTW + 2 * wr, gh = kRecTH + 2 * hr, x0 = blockIdx.x * kRecTW, y0 = blockIdx.y * kRecTH;
    if (want_code) {
        const int lane = threadIdx.x & 31;
        for (int r = threadIdx.x >> 5; r < gh; r += kRecT / 32) {
            // past the last pixel's window: clamped into range, never used
            const uint8_t *row = gray + (size_t)wrap1(imin(y0 - hr + r, H - 1 + hr), H) * W;
            uint8_t g[4];  // the row's (at most 64 + 2 * 31) columns in flight together
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int c = lane + 32 * k;
                g[k] = c < gw ? row[wrap1(imin(x0 - wr + c, W - 1 + wr), W)] : (uint8_t)0;
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (lane + 32 * k < gw) gt[r * gw + lane + 32 * k] = g[k];
        }
        __syncthreads();
    }
    const int px = threadIdx.x & (kRecTW - 1), x = x0 + px;
    if (x >= W) return;
    for (int py = threadIdx.x / kRecTW; py < kRecTH; py += kRecT / kRecTW) {
        const int y = y0 + py;
        if (y >= H) return;
        uint32_t lo = 0, hi = 0;
        if (want_code) {
            // seq/CensusTransform.cpp:11-37: strict centre > neighbour
            const uint8_t *g0 = gt + py * gw + px;
            const uint32_t c = g0[hr * gw + wr];
            if constexpr (WIN) {
#pragma unroll
                for (int r = 0; r < 9; r++)
#pragma unroll
                    for (int dx = 0; dx < 7; dx++) {
                        const uint32_t below = (uint32_t)g0[r * gw + dx] - c;  // sign bit: c > neighbour
                        if (7 * r + dx < 32) lo = __funnelshift_l(below, lo, 1);
                        else hi = __funnelshift_l(below, hi, 1);
                    }
            } else {
                int k = 0;
                for (int r = 0; r <= 2 * hr; r++)
                    for (int dx = 0; dx <= 2 * wr; dx++, k++) {
                        const uint32_t bit = c > (uint32_t)g0[r * gw + dx] ? 1u : 0u;
                        if (k < 32) lo |= bit << k;
                        else hi |= bit << (k - 32);
                    }
            }
        }
        const size_t p = (size_t)y * W + x;
        // without a colour image the gray in all three channels (seq/Main.cpp:87-90)
        const uint8_t *q = rgb + 3 * p;
        rec[p] = make_uint4(lo, hi,
                            rgb ? (uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16) : gray[p] * 0x010101u,
                            0u);
    }
}

// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_cost_volume(const uint4 *__restrict__ rr, const uint4 *__restrict__ rt, T *__restrict__ vol, int H,
                              int W, int D, int pitch, int mirror, CostCfg cfg) {
    const int y = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * D) return;
    const int x = i / D, d = i - x * D;
    const int xt = tar_col(x, d, W, 1);
    const uint4 a = rr[(size_t)y * W + (mirror ? W - 1 - x : x)], b = rt[(size_t)y * W + (mirror ? W - 1 - xt : xt)];
    vol[((size_t)y * W + x) * pitch + d] = to_store<T>(pair_cost(a, b, cfg));
}

// AD (optionally truncated) + census combined through the two host tables, the integer
// path.  Resident blocks stride over (row, 64 pixels); an item's reference records and the
// target records it meets, columns x0 - Dp .. x0 + 63 (wrapped as in
// seq/PixelBasedCost.cpp:19-20; Dp = D up to a multiple of 4), are staged in shared memory,
// target u in array u mod 4, so that a thread's 4 pixels x 4 disparities read 7 target
// records for 16 entries, lanes (disparity groups) on consecutive ones.  The tables are
// staged 2^lc1 and 2^lc2 times over, copy = lane: a warp's 32 lookups of one table hit
// nearly 32 different banks (a single copy costs some 3.5 wavefronts a lookup).
// Bound: the L1/shared data pipe (70 % busy: about 6 wavefronts a warp's 32 entries, records
// 2.75, lookups and their conflicts 3.5); the next item's records are fetched under the
// entries' work (1920x1080, D = 128, records and both volumes 608 -> 545 us).
constexpr int kAdcTX = 64;
constexpr int kAdcL1 = 768, kAdcL2 = 68;    // table entries staged: AD <= 765, census <= 64
constexpr int kAdcNT = (kAdcTX + 256) / 4;  // target records of one residue
static_assert(kAdcL1 * 16 * 4 + kAdcL2 * 32 * 4 + (4 * kAdcNT + kAdcTX) * 16 <= 75 * 1024, "three blocks an SM");

template <typename T>
__global__ void __launch_bounds__(256, 3) k_cost_volume_adc(const uint4 *__restrict__ rr, const uint4 *__restrict__ rt,
                                                           T *__restrict__ vol, int H, int W, int D, int pitch,
                                                           int mirror, int itrunc, const float *__restrict__ lut1,
                                                           const float *__restrict__ lut2, int lc1, int lc2) {
    extern __shared__ __align__(16) unsigned char asm2_[];
    uint4 *trec = reinterpret_cast<uint4 *>(asm2_), *rrec = trec + 4 * kAdcNT;  // [u mod 4][u / 4]; [64]
    float *t1 = reinterpret_cast<float *>(rrec + kAdcTX), *t2 = t1 + (kAdcL1 << lc1);
    const int tid = threadIdx.x, lane = tid & 31;
    for (int i = tid; i < kAdcL1 << lc1; i += 256) t1[i] = lut1[i >> lc1];
    for (int i = tid; i < kAdcL2 << lc2; i += 256) t2[i] = lut2[i >> lc2];
    const float *l1 = t1 + (lane & ((1 << lc1) - 1)), *l2 = t2 + (lane & ((1 << lc2) - 1));
    const int ndg = (D + 3) >> 2, Dp = 4 * ndg, xb = (W + kAdcTX - 1) / kAdcTX;
    const bool vec = (pitch & 3) == 0;
    // an item's records, two a thread (kAdcTX + Dp targets, then the references): fetched
    // while the previous item is worked
    static_assert(2 * kAdcTX + 256 <= 2 * 256, "two records a thread");
    uint4 next[2];
    auto fetch = [&](int item) {
        const int y = item / xb, x0 = (item - y * xb) * kAdcTX;
        const size_t row = (size_t)y * W;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int i = tid + 256 * k, ir = i - (kAdcTX + Dp);
            if (ir >= kAdcTX) continue;
            int x = x0 + (ir < 0 ? i - Dp : ir);
            if (x < 0) x += W;  // seq/PixelBasedCost.cpp:19-20 (D <= W)
            x = imax(imin(x, W - 1), 0);  // clamped: of no entry
            next[k] = (ir < 0 ? rt : rr)[row + (mirror ? W - 1 - x : x)];
        }
    };
    if ((int)blockIdx.x < H * xb) fetch(blockIdx.x);
    for (int item = blockIdx.x; item < H * xb; item += gridDim.x) {
        const int y = item / xb, x0 = (item - y * xb) * kAdcTX;
        const size_t row = (size_t)y * W;
        __syncthreads();  // the previous item's records are consumed (and the tables are in)
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int i = tid + 256 * k, ir = i - (kAdcTX + Dp);
            if (ir < 0) trec[(i & 3) * kAdcNT + (i >> 2)] = next[k];
            else if (ir < kAdcTX) rrec[ir] = next[k];
        }
        __syncthreads();
        if (item + (int)gridDim.x < H * xb) fetch(item + gridDim.x);
        const int nx = imin(kAdcTX, W - x0);
        // pixel group xg = q / ndg, disparity group dg = q mod ndg; 256 groups at a time
        const int sx = 256 / ndg, sd = 256 - sx * ndg;
        for (int xg = tid / ndg, dg = tid - xg * ndg; 4 * xg < nx;) {
            const uint4 *tb = trec + (xg - dg + ndg);  // u = 4 (xg - dg) + Dp + j - i
            uint4 b[7];                                // j - i + 3
#pragma unroll
            for (int k = 0; k < 7; k++) b[k] = k < 3 ? tb[(k + 1) * kAdcNT - 1] : tb[(k - 3) * kAdcNT];
            T *out = vol + (row + x0 + 4 * xg) * pitch + 4 * dg;
#pragma unroll
            for (int j = 0; j < 4; j++, out += pitch) {
                const uint4 a = rrec[4 * xg + j];
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint4 &t = b[j - i + 3];
                    const int sad = imin((int)__vsadu4(a.z, t.z), itrunc);   // seq/PixelBasedCost.cpp:86-91 / :106-112
                    const int ham = __popc(a.x ^ t.x) + __popc(a.y ^ t.y);  // seq/CensusTransform.cpp:52-60
                    v[i] = __fadd_rn(l1[sad << lc1], l2[ham << lc2]);       // seq/CombineCost.cpp:23
                }
                if (4 * xg + j < nx) {
                    if (vec) {
                        // (a padded pitch takes the cells past D too)
                        if constexpr (sizeof(T) == 4) {
                            *reinterpret_cast<float4 *>(out) = make_float4(v[0], v[1], v[2], v[3]);
                        } else {
                            const __half2 h0 = __floats2half2_rn(v[0], v[1]), h1 = __floats2half2_rn(v[2], v[3]);
                            *reinterpret_cast<uint2 *>(out) = make_uint2(*reinterpret_cast<const uint32_t *>(&h0),
                                                                         *reinterpret_cast<const uint32_t *>(&h1));
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            if (4 * dg + i < D) out[i] = to_store<T>(v[i]);
                    }
                }
            }
            xg += sx;
            dg += sd;
            if (dg >= ndg) {
                dg -= ndg;
                xg++;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Adaptive-weight aggregation fused with the arg-min.  Block: one row y, 64
// pixels x0..x0+63, all disparities in chunks of 64; 256 threads, each with
// 4 pixels x 4 disparities.  Warp w owns pixels 8w..8w+7 for all 64
// disparities (lane = 2 pixel groups x 16 disparity groups), so the reference
// weights are broadcast loads and the target weights and costs are contiguous.
// Per tap row ky the block stages the cost rows (wrapped columns x0-r ..
// x0+63+r), the packed Lab rows of the tap row, then the reference weights
// wR(p, ky, kx) and the target weights wT(t, ky, kx) for t = x0-dc0-63 ..
// x0-dc0+63 (wrapped), then every thread adds its 32 chains in the reference's
// order (plain form):
//   w = wR*wT;  sw = sw + w;  sc = sc + C*w      (seq/AdaptiveWeightAggregation.cpp:100-103)
// Tap rows outside the image have all-zero weights and add exact zeros, so
// they are skipped.  A weight is pw[k] * G[|Lab(p)-Lab(q)|^2] with host tables
// (seq/AdaptiveWeightAggregation.cpp:60-63); |Lab(p)-Lab(q)|^2 is the dot
// product of the byte-wise absolute differences of the packed Lab words.
constexpr int kAwTX = 64, kAwDC = 64, kAwThreads = 256;
constexpr int kAwCPitch = kAwDC + 4;
constexpr int kAwHPitch = kAwDC + 8;  // f16 cost rows: 144 bytes, a multiple of 16
constexpr uint32_t kLabOut = 0xff000000u;  // marks a column outside the image

__global__ void k_pack_lab(const uint8_t *__restrict__ lab, uint32_t *__restrict__ out, int W, int mirror) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= W) return;
    const size_t row = (size_t)blockIdx.y * W;
    const uint8_t *q = lab + 3 * (row + (mirror ? W - 1 - x : x));
    out[row + x] = (uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16);
}

template <typename CT, bool EXACT>
__global__ void __launch_bounds__(kAwThreads, 3) k_aw_wta(const CT *__restrict__ vol, const uint32_t *__restrict__ labr,
                                                      const uint32_t *__restrict__ labt, const float *__restrict__ pw,
                                                      const float *__restrict__ G, uint16_t *__restrict__ raw,
                                                      int *__restrict__ row_last, float *__restrict__ cost_out, int H,
                                                      int W, int D, int e) {
    // EXACT: the reference's unfused w*C then add (plain form); otherwise one fma
    const int r = e >> 1;
    constexpr int NT = kAwTX + kAwDC - 1;  // target columns of a tile
    constexpr int NTP = NT + 1;
    extern __shared__ __align__(16) float asm_[];
    float *Cs = asm_;                                   // [(64+2r+4)][kAwCPitch], 4 spare rows
    float *wRs = Cs + (kAwTX + 2 * r + 4) * kAwCPitch;  // [e][64]
    float *wTs = wRs + e * kAwTX;                       // [e][NTP]
    uint32_t *labRrow = reinterpret_cast<uint32_t *>(wTs + e * NTP);  // [64 + 2r]
    uint32_t *labTrow = labRrow + (kAwTX + 2 * r);                    // [NT + 2r]
    __shared__ float best_v[kAwTX];
    __shared__ int best_i[kAwTX];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int td = lane & 15;                      // disparities 4td .. 4td+3 of the chunk
    const int px0 = 8 * warp + 4 * (lane >> 4);  // pixels px0 .. px0+3 of the tile
    const int y = blockIdx.y, x0 = blockIdx.x * kAwTX;
    if (tid < kAwTX) {
        best_v[tid] = __int_as_float(0x7f800000);
        best_i[tid] = 0x7fffffff;
    }
    const bool vec = (D & 3) == 0;

    for (int dc0 = 0; dc0 < D; dc0 += kAwDC) {
        // sums of disparity pairs (4td + 2h, 4td + 2h + 1) of pixel px0 + j, packed for
        // the f32x2 instructions (each half an IEEE round-to-nearest operation)
        unsigned long long sw[4][2], sc[4][2];
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) sw[j][h] = sc[j][h] = 0ull;
        // centre Lab words: reference pixels x0+lane+32m, target columns t(u), u = lane+32m
        const int tbase = x0 - dc0 - (kAwDC - 1);  // target column of u = 0, before wrapping
        uint32_t cR[2], cT[4];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int x = x0 + lane + 32 * m;
            cR[m] = x < W ? labr[(size_t)y * W + x] : kLabOut;
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
            int t = tbase + lane + 32 * m;
            if (t < 0) t += W;  // seq/AdaptiveWeightAggregation.cpp:87
            cT[m] = (lane + 32 * m < NT && t >= 0 && t < W) ? labt[(size_t)y * W + t] : kLabOut;
        }
        // targets that wrapped around the left edge take their tap row from the
        // other end of the row; only tiles with tbase < 0 have them
        const bool wrapped_tile = tbase < 0;

        const int ky_lo = imax(-r, -y), ky_hi = imin(r, H - 1 - y);
        for (int ky = ky_lo; ky <= ky_hi; ky++) {
            const int yy = y + ky;
            __syncthreads();  // previous tap row fully consumed
            // cost rows, wrapped columns (seq/AdaptiveWeightAggregation.cpp:95-97); real pixels
            // wrap once (r < W), columns of padding pixels past the image end are clamped
            const size_t crow = (size_t)yy * W;
            if (vec) {
                for (int q = tid; q < (kAwTX + 2 * r) * (kAwDC / 4); q += kAwThreads) {
                    const int xi = q >> 4, d4 = (q & 15) * 4;
                    const int xs = imin(imax(wrap1(x0 - r + xi, W), 0), W - 1);
                    const int dg = dc0 + d4;
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (dg < D) {
                        const CT *src = vol + (crow + xs) * D + dg;
                        if constexpr (sizeof(CT) == 4) {
                            v = *reinterpret_cast<const float4 *>(src);
                        } else {
                            const uint2 hv = *reinterpret_cast<const uint2 *>(src);
                            const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&hv.x));
                            const float2 f1 = __half22float2(*reinterpret_cast<const __half2 *>(&hv.y));
                            v = make_float4(f0.x, f0.y, f1.x, f1.y);
                        }
                    }
                    *reinterpret_cast<float4 *>(Cs + xi * kAwCPitch + d4) = v;
                }
            } else {
                for (int q = tid; q < (kAwTX + 2 * r) * kAwDC; q += kAwThreads) {
                    const int xi = q >> 6, dd = q & 63;
                    const int xs = imin(imax(wrap1(x0 - r + xi, W), 0), W - 1);
                    const int dg = dc0 + dd;
                    Cs[xi * kAwCPitch + dd] = (dg < D) ? to_f32(vol[(crow + xs) * D + dg]) : 0.f;
                }
            }
            // packed Lab of the tap row: reference columns x0-r .., target columns tbase-r ..
            for (int q = tid; q < kAwTX + 2 * r; q += kAwThreads) {
                const int xc = x0 - r + q;
                labRrow[q] = (xc >= 0 && xc < W) ? labr[crow + xc] : kLabOut;
            }
            for (int q = tid; q < NT + 2 * r; q += kAwThreads) {
                const int xc = tbase - r + q;
                labTrow[q] = (xc >= 0 && xc < W) ? labt[crow + xc] : kLabOut;
            }
            __syncthreads();
            const float *pwrow = pw + (ky + r) * e;
            // weights of two taps per pass (kx and kx + 8), the table reads of both in
            // flight together: the colour-distance index of every weight first, then the
            // reads, then the products
            for (int kx = warp; kx < e; kx += 2 * (kAwThreads / 32)) {
                uint32_t idx[2][6];
                bool ok[2][6];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int k = kx + h * (kAwThreads / 32);
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        const uint32_t q = labRrow[imin(lane + 32 * m + k, kAwTX + 2 * r - 1)];
                        ok[h][m] = k < e && !((q | cR[m]) & kLabOut);
                        const uint32_t ad = __vabsdiffu4(cR[m], q);
                        idx[h][m] = __dp4a(ad, ad, 0u);
                    }
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        const int u = lane + 32 * m;
                        uint32_t q = labTrow[imin(u + k, NT + 2 * r - 1)];
                        if (wrapped_tile && tbase + u < 0 && k < e) {
                            // the target column is t + W: its tap is column t + W + k - r
                            const int xc = tbase + u + W + k - r;
                            q = (xc >= 0 && xc < W) ? labt[crow + xc] : kLabOut;
                        }
                        ok[h][2 + m] = k < e && u < NT && !((q | cT[m]) & kLabOut);
                        const uint32_t ad = __vabsdiffu4(cT[m], q);
                        idx[h][2 + m] = __dp4a(ad, ad, 0u);
                    }
                }
                float g[2][6];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int m = 0; m < 6; m++) g[h][m] = ok[h][m] ? __ldg(G + idx[h][m]) : 0.f;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int k = kx + h * (kAwThreads / 32);
                    if (k < e) {
                        // seq/AdaptiveWeightAggregation.cpp:33-71: pw[k] * expf(-dist / gamma_s),
                        // 0 where the tap (or a padding centre) is outside the image
                        const float pwk = __ldg(pwrow + k);
#pragma unroll
                        for (int m = 0; m < 2; m++) wRs[k * kAwTX + lane + 32 * m] = ok[h][m] ? __fmul_rn(pwk, g[h][m]) : 0.f;
#pragma unroll
                        for (int m = 0; m < 4; m++) {
                            const int u = lane + 32 * m;
                            if (u < NT) wTs[k * NTP + u] = ok[h][2 + m] ? __fmul_rn(pwk, g[h][2 + m]) : 0.f;
                        }
                    }
                }
            }
            __syncthreads();

            // u index of wT for (j, i): px0 + j - 4td - i + 63 = ubase + (j - i) + 3
            const int ubase = px0 - 4 * td + kAwDC - 4;
            const float *cp = Cs + px0 * kAwCPitch + 4 * td;  // cost column px0 + kx, + kx * pitch
            const float *wrp = wRs + px0;                      // + kx * 64
            const float *wtp = wTs + ubase;                    // + kx * NTP
            // one tap: 4 pixels x 4 disparities, reference order per entry
            auto tap = [&](const float (*cw)[4], int cofs, const float *wr4, const float *wt7) {
                float wr[4], wt[7];
                const float4 a0 = *reinterpret_cast<const float4 *>(wr4);
                wr[0] = a0.x; wr[1] = a0.y; wr[2] = a0.z; wr[3] = a0.w;
                const float4 b0 = *reinterpret_cast<const float4 *>(wt7);
                const float4 b1 = *reinterpret_cast<const float4 *>(wt7 + 4);
                wt[0] = b0.x; wt[1] = b0.y; wt[2] = b0.z; wt[3] = b0.w;
                wt[4] = b1.x; wt[5] = b1.y; wt[6] = b1.z;
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        // w of disparities i = 2h, 2h+1: wR * wT (index j - i + 3)
                        const unsigned long long w = pack2(__fmul_rn(wr[j], wt[j - 2 * h + 3]),
                                                           __fmul_rn(wr[j], wt[j - 2 * h + 2]));
                        const unsigned long long c = pack2(cw[j + cofs][2 * h], cw[j + cofs][2 * h + 1]);
                        sw[j][h] = add2(sw[j][h], w);
                        if constexpr (EXACT) sc[j][h] = add2(sc[j][h], mul2(c, w));
                        else sc[j][h] = fma2(c, w, sc[j][h]);
                    }
            };
            int kx = 0;
            // taps in groups of 4: the 7 cost columns px0+kx .. px0+kx+6 of a group are
            // loaded once and serve 4 pixels x 4 taps
#pragma unroll 1
            for (; kx + 4 <= e; kx += 4, cp += 4 * kAwCPitch, wrp += 4 * kAwTX, wtp += 4 * NTP) {
                float cw[7][4];
#pragma unroll
                for (int q = 0; q < 7; q++) {
                    const float4 v = *reinterpret_cast<const float4 *>(cp + q * kAwCPitch);
                    cw[q][0] = v.x; cw[q][1] = v.y; cw[q][2] = v.z; cw[q][3] = v.w;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) tap(cw, u, wrp + u * kAwTX, wtp + u * NTP);
            }
#pragma unroll 1
            for (; kx < e; kx++, cp += kAwCPitch, wrp += kAwTX, wtp += NTP) {
                float cw[4][4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float4 v = *reinterpret_cast<const float4 *>(cp + q * kAwCPitch);
                    cw[q][0] = v.x; cw[q][1] = v.y; cw[q][2] = v.z; cw[q][3] = v.w;
                }
                tap(cw, 0, wrp, wtp);
            }
        }
        __syncthreads();
        // score / sum of weights (seq/AdaptiveWeightAggregation.cpp:108), staged for the arg-min
        float *outs = Cs;  // [64][kAwDC + 1]
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float v = __fdiv_rn(half2_of(sc[j][i >> 1], i & 1), half2_of(sw[j][i >> 1], i & 1));
                outs[(px0 + j) * (kAwDC + 1) + 4 * td + i] = v;
                const int x = x0 + px0 + j, dg = dc0 + 4 * td + i;
                if (cost_out && x < W && dg < D) cost_out[((size_t)y * W + x) * D + dg] = v;
            }
        __syncthreads();
        if (tid < kAwTX) {
            float bv = best_v[tid];
            int bx = best_i[tid];
            const int nd = imin(kAwDC, D - dc0);
            for (int dd = 0; dd < nd; dd++) {
                const float v = outs[tid * (kAwDC + 1) + dd];
                if (v < bv) {  // first strict minimum in increasing d
                    bv = v;
                    bx = dc0 + dd;
                }
            }
            best_v[tid] = bv;
            best_i[tid] = bx;
        }
    }
    if (tid < kAwTX && x0 + tid < W) {
        const int x = x0 + tid;
        const bool found = best_i[tid] != 0;
        raw[(size_t)y * W + x] = found ? (uint16_t)(0x100 | best_i[tid]) : (uint16_t)0;
        if (found) atomicMax(row_last + y, x);
    }
}

// ---------------------------------------------------------------------------
// k_aw_wta, software-pipelined over the tap rows: while the
// block adds tap row ky, the cost rows of ky + 1 arrive by cp.async in the
// other buffer, the weights of ky + 1 are made in slices between the groups of
// taps (their table reads in flight across a group), and the Lab rows of
// ky + 2 are staged; one barrier per tap row.  The arithmetic per entry is
// k_aw_wta's: EXACT (plain form, f32 volume) the reference's order, unfused;
// otherwise (FP16 form, f16 volume staged as f16, a pitch that is a multiple of 8) one
// FMA.  pitch: values from pixel to pixel of the volume, at least D; cells past D belong to
// no disparity, and the sums they enter are dropped.
// E: the window edge as a constant (33, the reference driver's 33 x 33 window), so
// that the tap loop unrolls whole, or 0 for the edge of the e argument.
__device__ int g_aw_tma_timeouts;
uint64_t aw_tma_timeouts() {
    int v = 0;
    return cudaMemcpyFromSymbol(&v, g_aw_tma_timeouts, sizeof(int)) == cudaSuccess ? (uint64_t)v : 0;
}

template <typename CT, bool EXACT, int E>
__global__ void __launch_bounds__(kAwThreads, 2) k_aw_wta_pipe(const __grid_constant__ CUtensorMap tmap, int use_tma,
                                                          const CT *__restrict__ vol,
                                                          const uint32_t *__restrict__ labr,
                                                          const uint32_t *__restrict__ labt,
                                                          const float *__restrict__ pw, const float *__restrict__ G,
                                                          uint16_t *__restrict__ raw, int *__restrict__ row_last,
                                                          float *__restrict__ cost_out, int H, int W, int D, int pitch, int e_arg,
                                                          float zero) {
    const int e = E ? E : e_arg;
    const int r = e >> 1;
    // zero: +0.0f from the host.  A packed multiply whose result feeds a packed add is
    // contracted into one fused multiply-add by the compiler, even written as
    // mul.rn / __fmul2_rn; a fused multiply-add with this zero as its addend (which
    // the compiler cannot know is zero) rounds like the multiply alone and is not
    // fused further, so the plain form's products C*w stay IEEE products, two to an
    // instruction.
    const float2 z2 = make_float2(zero, zero);
    constexpr int NT = kAwTX + kAwDC - 1;  // target columns of a tile
    constexpr int NTP = NT + 1;
    // cost rows: 64 floats (dense, as a TMA copy writes them), or kAwHPitch halves
    // (16-byte rows for the copies, the pitch keeping a half warp's rows apart in banks)
    constexpr int CP = sizeof(CT) == 4 ? kAwDC : kAwHPitch;
    const int CS = (kAwTX + 2 * r + 4) * CP * (int)sizeof(CT) / 4;  // floats of one cost buffer
    // no static shared memory: the dynamic buffers begin at the block's shared base,
    // which the TMA copies need 128-byte aligned (checked per block; blocks whose
    // base is not take cp.async).  The declaration promises only 16 bytes, the
    // alignment the compiler's address arithmetic was tuned under.
    extern __shared__ __align__(16) float psm_[];
    // buffer b: costs at psm_ + b CS, reference weights at wR0 + b e 64, target weights at wT0 + b e NTP
    float *const wR0 = psm_ + 2 * CS, *const wT0 = wR0 + 2 * e * kAwTX;
    uint32_t *labbase = reinterpret_cast<uint32_t *>(psm_ + 2 * CS + 2 * e * kAwTX + 2 * e * NTP);
    const int LRN = kAwTX + 2 * r, LTN = NT + 2 * r;  // words of a reference / target Lab row
    float *const best_v = reinterpret_cast<float *>(labbase + 3 * (LRN + LTN));  // [kAwTX]
    int *const best_i = reinterpret_cast<int *>(best_v + kAwTX);                  // [kAwTX]
    // plain form, tiles whose cost columns need no wrap: each tap row's cost rows arrive
    // by one TMA copy (box 64 disparities x (64 + 2r) columns) completing on cbar[buffer]
    uint64_t *const cbar =
        reinterpret_cast<uint64_t *>((reinterpret_cast<uintptr_t>(best_i + kAwTX) + 7) & ~uintptr_t(7));  // [2]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = kAwThreads / 32;
    // tap tile: warp (wx, wd) = (warp & 3, warp >> 2) takes pixels 16 wx .. 16 wx + 15 and
    // disparities 32 wd .. 32 wd + 31 of the tile; lane (pg, dg) = (lane >> 3, lane & 7)
    // four pixels px0 .. px0+3 and four disparities dd0 .. dd0+3 of those.  Per tap a
    // warp reads 4 distinct reference weights, 11 distinct 16-byte target-weight
    // runs and one new cost column of 32 x 4 values (the other three of a thread's
    // window are in registers from the previous taps).
    const int px0 = 16 * (warp & 3) + 4 * (lane >> 3);
    const int dd0 = 32 * (warp >> 2) + 4 * (lane & 7);
    const int y = blockIdx.y, x0 = blockIdx.x * kAwTX;
    if (tid < kAwTX) {
        best_v[tid] = __int_as_float(0x7f800000);
        best_i[tid] = 0x7fffffff;
    }
    const bool vec = (pitch & 3) == 0;
    const bool tma_tile = sizeof(CT) == 4 && use_tma && x0 - r >= 0 && x0 + kAwTX + r <= W &&
                          ((uint32_t)__cvta_generic_to_shared(psm_) & 127) == 0;
    const uint32_t cb0 = (uint32_t)__cvta_generic_to_shared(cbar);
    uint32_t cphase = 0;  // bit b: parity of the next completion of cbar[b]
    if (tma_tile && tid == 0) {
        mbar_init(cb0);
        mbar_init(cb0 + 8);
    }
    // (the barriers' initialisation is published by the chunk loop's first __syncthreads)
    auto cost_wait = [&](int b) {
        if (!tma_tile) return;
        if (!mbar_wait(cb0 + 8 * b, (cphase >> b) & 1)) {
            if (tid == 0) atomicAdd(&g_aw_tma_timeouts, 1);
            mbar_wait(cb0 + 8 * b, (cphase >> b) & 1);  // the copy may still land in this buffer
        }
        cphase ^= 1u << b;
    };

    for (int dc0 = 0; dc0 < D; dc0 += kAwDC) {
        // sums of disparity pairs (dd0 + 2h, dd0 + 2h + 1) of pixel px0 + j, as float2 for
        // the packed adds (each half an IEEE round-to-nearest operation)
        float2 sw[4][2], sc[4][2];
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) sw[j][h] = sc[j][h] = make_float2(0.f, 0.f);
        const int tbase = x0 - dc0 - (kAwDC - 1);
        uint32_t cR[2], cT[4];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int x = x0 + lane + 32 * m;
            cR[m] = x < W ? labr[(size_t)y * W + x] : kLabOut;
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
            int t = tbase + lane + 32 * m;
            if (t < 0) t += W;  // seq/AdaptiveWeightAggregation.cpp:87
            cT[m] = (lane + 32 * m < NT && t >= 0 && t < W) ? labt[(size_t)y * W + t] : kLabOut;
        }
        const bool wrapped_tile = tbase < 0;
        const int ky_lo = imax(-r, -y), ky_hi = imin(r, H - 1 - y);

        // cost rows of tap row ky into C by cp.async (zero fill past D); wrapped
        // columns as in k_aw_wta (seq/AdaptiveWeightAggregation.cpp:95-97)
        auto stage_cost = [&](int ky, int b) {
            float *C = psm_ + b * CS;
            const size_t crow = (size_t)(y + ky) * W;
            const uint32_t cbase = (uint32_t)__cvta_generic_to_shared(C);
            if (tma_tile) {
                if (tid == 0)
                    tma_load_3d(cbase, &tmap, dc0, x0 - r, y + ky, cb0 + 8 * b,
                                (uint32_t)((kAwTX + 2 * r) * kAwDC * sizeof(float)));
                return;
            }
            if constexpr (sizeof(CT) == 2) {
                // f16 volume: 16-byte copies of 8 disparities (the pitch is a multiple of 8)
                for (int q = tid; q < (kAwTX + 2 * r) * (kAwDC / 8); q += kAwThreads) {
                    const int xi = q >> 3, d8 = (q & 7) * 8;
                    const int xs = imin(imax(wrap1(x0 - r + xi, W), 0), W - 1);
                    const int dg = dc0 + d8;
                    const CT *src = vol + (crow + xs) * pitch + (dg < D ? dg : 0);
                    const uint32_t dst = cbase + (uint32_t)((xi * CP + d8) * 2);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
                                 "r"(dg < D ? 16 : 0)
                                 : "memory");
                }
            } else if (vec) {
                for (int q = tid; q < (kAwTX + 2 * r) * (kAwDC / 4); q += kAwThreads) {
                    const int xi = q >> 4, d4 = (q & 15) * 4;
                    const int xs = imin(imax(wrap1(x0 - r + xi, W), 0), W - 1);
                    const int dg = dc0 + d4;
                    const float *src = vol + (crow + xs) * pitch + (dg < D ? dg : 0);
                    const uint32_t dst = cbase + (uint32_t)((xi * CP + d4) * 4);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
                                 "r"(dg < D ? 16 : 0)
                                 : "memory");
                }
            } else {
                for (int q = tid; q < (kAwTX + 2 * r) * kAwDC; q += kAwThreads) {
                    const int xi = q >> 6, dd = q & 63;
                    const int xs = imin(imax(wrap1(x0 - r + xi, W), 0), W - 1);
                    const int dg = dc0 + dd;
                    const float *src = vol + (crow + xs) * pitch + (dg < D ? dg : 0);
                    const uint32_t dst = cbase + (uint32_t)((xi * CP + dd) * 4);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src),
                                 "r"(dg < D ? 4 : 0)
                                 : "memory");
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        auto stage_lab = [&](int ky, int slot) {
            const size_t crow = (size_t)(y + ky) * W;
            uint32_t *LR = labbase + slot * (LRN + LTN), *LT = LR + LRN;
            for (int q = tid; q < LRN; q += kAwThreads) {
                const int xc = x0 - r + q;
                LR[q] = (xc >= 0 && xc < W) ? labr[crow + xc] : kLabOut;
            }
            for (int q = tid; q < LTN; q += kAwThreads) {
                const int xc = tbase - r + q;
                LT[q] = (xc >= 0 && xc < W) ? labt[crow + xc] : kLabOut;
            }
        };
        // weights of tap (ky, k) for this warp's lanes, in two halves: the table
        // indices and reads (issue), then the products (finish)
        struct Slice {
            uint32_t idx[6];
            bool ok[6];
            float g[6];
        };
        // (every caller passes k < e, so the reference index lane + 32 m + k <= 63 + 2r
        // stays inside its row, and the target index u + k only passes the row's end
        // for u = 127, the padding target of lane 31)
        auto slice_issue = [&](Slice &sl, int ky, int k, int slot) {
            const uint32_t *LR = labbase + slot * (LRN + LTN), *LT = LR + LRN;
#pragma unroll
            for (int m = 0; m < 2; m++) {
                const uint32_t q = LR[lane + 32 * m + k];
                sl.ok[m] = !((q | cR[m]) & kLabOut);
                const uint32_t ad = __vabsdiffu4(cR[m], q);
                sl.idx[m] = __dp4a(ad, ad, 0u);
            }
            uint32_t qt[4];
#pragma unroll
            for (int m = 0; m < 3; m++) qt[m] = LT[lane + 32 * m + k];
            qt[3] = LT[imin(lane + 96 + k, LTN - 1)];
            if (wrapped_tile) {
                // targets that wrapped around the left edge: their taps come from the
                // other end of the row (block-uniform branch)
                const size_t crow = (size_t)(y + ky) * W;
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    const int u = lane + 32 * m;
                    if (tbase + u < 0) {
                        const int xc = tbase + u + W + k - r;
                        qt[m] = (xc >= 0 && xc < W) ? labt[crow + xc] : kLabOut;
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < 4; m++) {
                sl.ok[2 + m] = (m < 3 || lane < 31) && !((qt[m] | cT[m]) & kLabOut);
                const uint32_t ad = __vabsdiffu4(cT[m], qt[m]);
                sl.idx[2 + m] = __dp4a(ad, ad, 0u);
            }
#pragma unroll
            for (int m = 0; m < 6; m++) sl.g[m] = sl.ok[m] ? __ldg(G + sl.idx[m]) : 0.f;
        };
        auto slice_finish = [&](const Slice &sl, int ky, int k, float *wR, float *wT) {
            if (k < e) {
                // seq/AdaptiveWeightAggregation.cpp:33-71: pw[k] * expf(-dist / gamma_s)
                const float pwk = __ldg(pw + (ky + r) * e + k);
#pragma unroll
                for (int m = 0; m < 2; m++) wR[k * kAwTX + lane + 32 * m] = sl.ok[m] ? __fmul_rn(pwk, sl.g[m]) : 0.f;
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    const int u = lane + 32 * m;
                    if (u < NT) wT[k * NTP + u] = sl.ok[2 + m] ? __fmul_rn(pwk, sl.g[2 + m]) : 0.f;
                }
            }
        };

        // prologue: Lab rows of the first two tap rows, costs and weights of the first
        __syncthreads();  // the previous chunk is done with every buffer
        stage_lab(ky_lo, 0);
        if (ky_lo + 1 <= ky_hi) stage_lab(ky_lo + 1, 1);
        stage_cost(ky_lo, 0);
        __syncthreads();
        for (int k = warp; k < e; k += NW) {
            Slice sl;
            slice_issue(sl, ky_lo, k, 0);
            slice_finish(sl, ky_lo, k, wR0, wT0);
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        cost_wait(0);
        __syncthreads();

        for (int ky = ky_lo; ky <= ky_hi; ky++) {
            const int i = ky - ky_lo, b = i & 1;
            const bool next = ky + 1 <= ky_hi;
            if (next) stage_cost(ky + 1, b ^ 1);
            if (ky + 2 <= ky_hi) stage_lab(ky + 2, (i + 2) % 3);
            const int lnext = (i + 1) % 3;
            const float *Cs = psm_ + b * CS, *wRs = wR0 + b * e * kAwTX, *wTs = wT0 + b * e * NTP;
            float *wRn = wR0 + (b ^ 1) * e * kAwTX, *wTn = wT0 + (b ^ 1) * e * NTP;

            // target weights of entry (j, i): u = px0 + j - (dd0 + i) + 63, so a thread's
            // seven are ub .. ub+6 (the eighth loaded is ub+7 <= 127, inside the row)
            const int ub = px0 - dd0 + kAwDC - 4;
            const CT *cp = reinterpret_cast<const CT *>(Cs) + px0 * CP + dd0;  // staged column px0 + kx
            const float *wrp = wRs + px0;
            const float *wtp = wTs + ub;
            // four disparities of a staged cost column as floats
            auto col4 = [&](const CT *q, float *o) {
                if constexpr (sizeof(CT) == 4) {
                    const float4 v = *reinterpret_cast<const float4 *>(q);
                    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
                } else {
                    const uint2 hv = *reinterpret_cast<const uint2 *>(q);
                    const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&hv.x));
                    const float2 f1 = __half22float2(*reinterpret_cast<const __half2 *>(&hv.y));
                    o[0] = f0.x; o[1] = f0.y; o[2] = f1.x; o[3] = f1.y;
                }
            };
            // one tap over the thread's 4 pixels x 4 disparities; cw[j] is the cost column
            // of pixel j at this tap.  Plain form (EXACT): w = wR*wT, sw += w, sc += C*w, each
            // an IEEE operation (seq/AdaptiveWeightAggregation.cpp:100-103): w by scalar
            // multiplies, C*w by the packed multiply-add with the opaque zero, the sums by
            // packed adds.  FP16 form: sc = fma(C, w, sc).
            auto tap = [&](const float (&cw)[4][4], const float *wr4, const float *wt8) {
                float wr[4], wt[8];
                const float4 a0 = *reinterpret_cast<const float4 *>(wr4);
                wr[0] = a0.x; wr[1] = a0.y; wr[2] = a0.z; wr[3] = a0.w;
                const float4 b0 = *reinterpret_cast<const float4 *>(wt8);
                const float4 b1 = *reinterpret_cast<const float4 *>(wt8 + 4);
                wt[0] = b0.x; wt[1] = b0.y; wt[2] = b0.z; wt[3] = b0.w;
                wt[4] = b1.x; wt[5] = b1.y; wt[6] = b1.z; wt[7] = b1.w;
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float w0 = __fmul_rn(wr[j], wt[j - 2 * h + 3]);
                        const float w1 = __fmul_rn(wr[j], wt[j - 2 * h + 2]);
                        sw[j][h] = __fadd2_rn(sw[j][h], make_float2(w0, w1));
                        if constexpr (EXACT)
                            sc[j][h] = __fadd2_rn(sc[j][h], __ffma2_rn(make_float2(cw[j][2 * h], cw[j][2 * h + 1]),
                                                                       make_float2(w0, w1), z2));
                        else
                            sc[j][h] = __ffma2_rn(make_float2(cw[j][2 * h], cw[j][2 * h + 1]), make_float2(w0, w1),
                                                  sc[j][h]);
                    }
            };
            // the cost window slides one column per tap: win holds columns kx .. kx+2 of
            // the thread's first pixel, each tap adds column kx+3
            float win[3][4];
#pragma unroll
            for (int q = 0; q < 3; q++) col4(cp + q * CP, win[q]);
            int kx = 0, sj = 0;
#pragma unroll(E ? 8 : 1)
            for (; kx + 4 <= e; kx += 4, sj++) {
                // a slice of the next tap row's weights around this group of taps
                const int ks = warp + NW * sj;
                const bool dos = next && ks < e;
                Slice sl;
                if (dos) slice_issue(sl, ky + 1, ks, lnext);
                float nc[4][4];
#pragma unroll
                for (int u = 0; u < 4; u++) col4(cp + (kx + 3 + u) * CP, nc[u]);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    float cw[4][4];
#pragma unroll
                    for (int j = 0; j < 4; j++)
#pragma unroll
                        for (int i = 0; i < 4; i++) cw[j][i] = (u + j < 3) ? win[u + j][i] : nc[u + j - 3][i];
                    tap(cw, wrp + (kx + u) * kAwTX, wtp + (kx + u) * NTP);
                }
#pragma unroll
                for (int q = 0; q < 3; q++)
#pragma unroll
                    for (int i = 0; i < 4; i++) win[q][i] = nc[q + 1][i];
                if (dos) slice_finish(sl, ky + 1, ks, wRn, wTn);
            }
#pragma unroll(E ? 3 : 1)
            for (; kx < e; kx++) {
                float cw[4][4];
                col4(cp + (kx + 3) * CP, cw[3]);
#pragma unroll
                for (int q = 0; q < 3; q++)
#pragma unroll
                    for (int i = 0; i < 4; i++) cw[q][i] = win[q][i];
                tap(cw, wrp + kx * kAwTX, wtp + kx * NTP);
#pragma unroll
                for (int q = 0; q < 3; q++)
#pragma unroll
                    for (int i = 0; i < 4; i++) win[q][i] = cw[q + 1][i];
            }
            // slices the groups did not reach (short windows)
            if (next)
                for (int ks = warp + NW * sj; ks < e; ks += NW) {
                    Slice sl;
                    slice_issue(sl, ky + 1, ks, lnext);
                    slice_finish(sl, ky + 1, ks, wRn, wTn);
                }
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            if (next) cost_wait(b ^ 1);
            __syncthreads();
        }
        // score / sum of weights (seq/AdaptiveWeightAggregation.cpp:108), staged for the arg-min
        float *outs = psm_;  // [64][kAwDC + 1]
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 a2 = sc[j][i >> 1], b2 = sw[j][i >> 1];
                const float v = __fdiv_rn((i & 1) ? a2.y : a2.x, (i & 1) ? b2.y : b2.x);
                outs[(px0 + j) * (kAwDC + 1) + dd0 + i] = v;
                const int x = x0 + px0 + j, dg = dc0 + dd0 + i;
                if (cost_out && x < W && dg < D) cost_out[((size_t)y * W + x) * D + dg] = v;
            }
        __syncthreads();
        if (tid < kAwTX) {
            float bv = best_v[tid];
            int bx = best_i[tid];
            const int nd = imin(kAwDC, D - dc0);
            for (int dd = 0; dd < nd; dd++) {
                const float v = outs[tid * (kAwDC + 1) + dd];
                if (v < bv) {  // first strict minimum in increasing d
                    bv = v;
                    bx = dc0 + dd;
                }
            }
            best_v[tid] = bv;
            best_i[tid] = bx;
        }
    }
    if (tid < kAwTX && x0 + tid < W) {
        const int x = x0 + tid;
        const bool found = best_i[tid] != 0;
        raw[(size_t)y * W + x] = found ? (uint16_t)(0x100 | best_i[tid]) : (uint16_t)0;
        if (found) atomicMax(row_last + y, x);
    }
}

// ---------------------------------------------------------------------------
// host orchestration

static bool fast_kind(int k) { return k == RTS_COST_AD || k == RTS_COST_CENSUS; }

bool fast_costs(const rts_params &p) {
    if (!fast_kind(p.cost1) || !(p.cost2 == RTS_COST_NONE || fast_kind(p.cost2))) return false;
    const bool census = p.cost1 == RTS_COST_CENSUS || p.cost2 == RTS_COST_CENSUS;
    return !census || (2 * p.census_hrad + 1) * (2 * p.census_wrad + 1) <= 64;
}

bool costs_nonneg(const rts_params &p) {
    if (p.cost1 == RTS_COST_NCC || p.cost2 == RTS_COST_NCC) return false;
    if (p.cost1 == RTS_COST_AD && p.aggr == RTS_AGGR_CROSS && !(p.ad_trunc >= 0.f)) return false;
    return p.cost2 == RTS_COST_NONE || (p.lambda1 > 0.f && p.lambda2 > 0.f);
}

bool fused_supported(const rts_params &p, int H, int W) {
    (void)H;
    (void)W;
    if (p.aggr == RTS_AGGR_CROSS) return cross_fused_supported(p);
    if (p.aggr == RTS_AGGR_AW) return p.aw_rad <= 16;
    return false;
}

rts_status prep_records(rts_ctx *c, const rts_params &p, int H, int W, const uint8_t *gray, const uint8_t *rgb,
                        uint4 *rec) {
    const int code = (p.cost1 == RTS_COST_CENSUS || p.cost2 == RTS_COST_CENSUS) && fast_costs(p) ? 1 : 0;
    const int hr = code ? p.census_hrad : 0, wr = code ? p.census_wrad : 0;
    const dim3 g((W + kRecTW - 1) / kRecTW, (H + kRecTH - 1) / kRecTH);
    const size_t smem = (size_t)(kRecTH + 2 * hr) * (kRecTW + 2 * wr);  // a window of at most 64 bits
    if (code && hr == 4 && wr == 3) k_prep_records<true><<<g, kRecT, smem, c->stream>>>(gray, rgb, rec, H, W, hr, wr, code);
    else k_prep_records<false><<<g, kRecT, smem, c->stream>>>(gray, rgb, rec, H, W, hr, wr, code);
    count_launch(c);
    return check_launch(c, "prep_records");
}

static rts_status cost_cfg(rts_ctx *c, const rts_params &p, CostCfg *cfg) {
    cfg->k1 = p.cost1;
    cfg->k2 = p.cost2;
    cfg->trunc1 = (p.cost1 == RTS_COST_AD && p.aggr == RTS_AGGR_CROSS) ? 1 : 0;  // seq/Main.cpp:183-186
    cfg->trunc = p.ad_trunc;
    cfg->l1 = p.lambda1;
    cfg->l2 = p.lambda2;
    cfg->lut1 = cfg->lut2 = nullptr;
    // integer fast path: AD with an integral truncation (or none) and census take
    // integer values below the table size (AD <= 765, census <= 64)
    const bool trunc_ok = !cfg->trunc1 || (p.ad_trunc >= 0.f && p.ad_trunc < (float)kCombineLut &&
                                          p.ad_trunc == floorf(p.ad_trunc));
    cfg->int_path = trunc_ok ? 1 : 0;
    cfg->itrunc = cfg->trunc1 ? (int)p.ad_trunc : 0x7fffffff;
    if (p.cost2 != RTS_COST_NONE) return combine_luts(c, p.lambda1, p.lambda2, &cfg->lut1, &cfg->lut2);
    return RTS_OK;
}

rts_status cost_volume_fast(rts_ctx *c, const rts_params &p, int H, int W, const uint4 *rr, const uint4 *rt,
                            void *vol, int half, int pitch, int mirror) {
    CostCfg cfg;
    RTS_TRY(cost_cfg(c, p, &cfg));
    const int D = p.disp_range;
    if (cfg.int_path && cfg.k1 == RTS_COST_AD && cfg.k2 == RTS_COST_CENSUS) {
        // copies of the tables where every resident block makes several items (staging 16 and 32
        // copies takes about one item's time)
        const long items = (long)((W + kAdcTX - 1) / kAdcTX) * H, res = 3L * sm_count();
        const int lc1 = items >= 4 * res ? 4 : 0, lc2 = items >= 4 * res ? 5 : 0;
        const size_t smem = ((size_t)(kAdcL1 << lc1) + (size_t)(kAdcL2 << lc2)) * 4 + (4 * kAdcNT + kAdcTX) * sizeof(uint4);
        auto go = [&](auto kern, auto *v) -> rts_status {
            RTS_TRY(set_smem(c, kern, smem, "cost_volume"));
            kern<<<(unsigned)std::min(items, lc1 ? res : items), 256, smem, c->stream>>>(
                rr, rt, v, H, W, D, pitch, mirror, cfg.itrunc, cfg.lut1, cfg.lut2, lc1, lc2);
            return RTS_OK;
        };
        if (half) RTS_TRY(go(k_cost_volume_adc<__half>, (__half *)vol));
        else RTS_TRY(go(k_cost_volume_adc<float>, (float *)vol));
        count_launch(c);
        return check_launch(c, "cost_volume");
    }
    const dim3 g((unsigned)(((long)W * D + 255) / 256), H);
    if (half) k_cost_volume<__half><<<g, 256, 0, c->stream>>>(rr, rt, (__half *)vol, H, W, D, pitch, mirror, cfg);
    else k_cost_volume<float><<<g, 256, 0, c->stream>>>(rr, rt, (float *)vol, H, W, D, pitch, mirror, cfg);
    count_launch(c);
    return check_launch(c, "cost_volume");
}

bool cross_fused_supported(const rts_params &p) {
    // the 64-entry ring of the horizontal kernel bounds the arm length (k_batch.cu); ranges
    // that are not a multiple of 8 go the way of cross_ragged_supported
    return p.cross_arm <= 23 && p.disp_range % 8 == 0;
}

bool cross_ragged_supported(const rts_params &p) {
    // The view kernels take any range, with the results of the composed module kernels
    // (450x375, D = 60, photo: 571 us a pair composed, 256 us here) where costs are made from records
    // and are >= 0 (their quotients take the fast exact division).  Other costs stay composed.
    return p.aggr == RTS_AGGR_CROSS && p.cross_arm <= 23 && p.disp_range % 8 != 0 && cross_record_costs(p) &&
           costs_nonneg(p);
}

rts_status aw_fused(rts_ctx *c, const rts_params &p, int H, int W, const void *vol, int half, int pitch, const uint8_t *labr,
                    const uint8_t *labt, int mirror, uint16_t *raw, int *rl, float *cost_out) {
    const float *pw, *g;
    RTS_TRY(prox_weights(c, p.aw_gamma_p, p.aw_rad, &pw));
    RTS_TRY(lab_weight_lut(c, p.aw_gamma_s, &g));
    const long np = (long)H * W;
    void *lp;
    RTS_TRY(scratch(c, SL_V_MEAN, (size_t)np * 8, &lp));
    uint32_t *plr = (uint32_t *)lp, *plt = plr + np;
    k_pack_lab<<<dim3((W + 255) / 256, H), 256, 0, c->stream>>>(labr, plr, W, mirror);
    k_pack_lab<<<dim3((W + 255) / 256, H), 256, 0, c->stream>>>(labt, plt, W, mirror);
    count_launch(c, 2);
    const int r = p.aw_rad, e = 2 * r + 1;
    const size_t smem = sizeof(float) * ((size_t)(kAwTX + 2 * r + 4) * kAwCPitch + (size_t)e * kAwTX +
                                         (size_t)e * (kAwTX + kAwDC) + (size_t)(kAwTX + 2 * r) +
                                         (size_t)(kAwTX + kAwDC - 1 + 2 * r));
    const dim3 grid((W + kAwTX - 1) / kAwTX, H);
    StageScope sc(c, "aw_wta");
    auto go = [&](auto kern, auto *v) -> rts_status {
        RTS_TRY(set_smem(c, kern, smem, "aw_wta"));
        kern<<<grid, kAwThreads, smem, c->stream>>>(v, plr, plt, pw, g, raw, rl, cost_out, H, W, p.disp_range, e);
        return RTS_OK;
    };
    // plain form: bit-exact float volume, the pipelined kernel; FP16 form: __half
    // volume and fused multiply-add
    // two cost buffers (their space also holds the [64][65] arg-min staging), two
    // weight buffers, three Lab row pairs, the arg-min state and two mbarriers
    auto pipe_smem = [&](size_t row_bytes) {
        const size_t costs = 2 * (size_t)(kAwTX + 2 * r + 4) * row_bytes;
        return std::max(costs, (size_t)kAwTX * (kAwDC + 1) * 4) +
               sizeof(float) * (2 * (size_t)e * kAwTX + 2 * (size_t)e * (kAwTX + kAwDC)) +
               sizeof(uint32_t) * 3 * ((size_t)(kAwTX + 2 * r) + (size_t)(kAwTX + kAwDC - 1 + 2 * r)) +
               2 * kAwTX * 4 + 24;
    };
    CUtensorMap tm{};
    if (half && pitch % 8 != 0) {
        RTS_TRY(go(k_aw_wta<__half, false>, (const __half *)vol));
    } else if (half) {
        const size_t psmem = pipe_smem((size_t)kAwHPitch * 2);
        auto kern = e == 33 ? k_aw_wta_pipe<__half, false, 33> : k_aw_wta_pipe<__half, false, 0>;
        RTS_TRY(set_smem(c, kern, psmem, "aw_wta_pipe"));
        kern<<<grid, kAwThreads, psmem, c->stream>>>(tm, 0, (const __half *)vol, plr, plt, pw, g, raw, rl, cost_out,
                                                     H, W, p.disp_range, pitch, e, 0.f);
    } else {
        // dense 64-float cost rows; the tiles whose columns need no wrap take them by TMA
        const size_t psmem = pipe_smem((size_t)kAwDC * 4);
        const int use_tma = volume_tensor_map(&tm, vol, H, W, p.disp_range, pitch, 4, kAwDC, kAwTX + 2 * r, 1) ? 1 : 0;
        auto kern = e == 33 ? k_aw_wta_pipe<float, true, 33> : k_aw_wta_pipe<float, true, 0>;
        RTS_TRY(set_smem(c, kern, psmem, "aw_wta_pipe"));
        kern<<<grid, kAwThreads, psmem, c->stream>>>(tm, use_tma, (const float *)vol, plr, plt, pw, g, raw, rl,
                                                     cost_out, H, W, p.disp_range, pitch, e, 0.f);
    }
    count_launch(c);
    return check_launch(c, "aw_wta");
}

}  // namespace rts
