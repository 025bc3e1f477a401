// k_aw_mod.cu -- adaptive support weights, module form
// (seq/AdaptiveWeightAggregation.cpp:33-150): weight arrays, and the aggregation of a
// cost volume by given weight arrays.
//
// Per entry the reference's arithmetic in its order, unfused (weight = wR wT, sums of
// weights and of C weight in raster order, their quotient).
#include <algorithm>

#include "rts_common.cuh"

namespace rts {

// ---------------------------------------------------------------------------
// Weight arrays: w[p][k] = pw[k] * G[|Lab(p)-Lab(q)|^2], 0 outside the image.  G is the
// host-computed expf(-sqrtf(n)/gamma_s), so the product is the reference's.

// any radius: a thread per weight
__global__ void k_compute_weights(const uint8_t *__restrict__ lab, const float *__restrict__ pw,
                                  const float *__restrict__ g, float *__restrict__ w, int H, int W, int r) {
    const int y = blockIdx.y;
    const int e = 2 * r + 1, area = e * e;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long)W * area) return;
    const int x = (int)(i / area), k = (int)(i - (long)x * area);
    const int dy = k / e - r, dx = k - (k / e) * e - r;
    const int yy = y + dy, xx = x + dx;
    float v = 0.f;
    if (yy >= 0 && yy < H && xx >= 0 && xx < W) {
        const uint8_t *a = lab + 3 * ((size_t)y * W + x);
        const uint8_t *b = lab + 3 * ((size_t)yy * W + xx);
        const int d0 = (int)a[0] - b[0], d1 = (int)a[1] - b[1], d2 = (int)a[2] - b[2];
        v = __fmul_rn(pw[k], g[d0 * d0 + d1 * d1 + d2 * d2]);
    }
    w[((size_t)y * W + x) * area + k] = v;
}

// Block per (row, kCwPx pixels): the packed Lab words of the pixels' windows staged in
// shared memory, a warp per pixel, lanes along the window (whole lines written).  Bound:
// the scattered reads of the 780 KB table (a thread per weight spent most of its time on
// three divisions and six byte loads: 240x180, 33x33 209 us an image; 62 us now).
constexpr int kCwPx = 16, kCwT = 256;
constexpr uint32_t kCwOut = 0xff000000u;  // marks a pixel outside the image
static size_t cw_smem(int r) { return (size_t)(2 * r + 1) * (kCwPx + 2 * r) * sizeof(uint32_t); }

__global__ void __launch_bounds__(kCwT) k_compute_weights_tile(const uint8_t *__restrict__ lab,
                                                              const float *__restrict__ pw,
                                                              const float *__restrict__ g, float *__restrict__ w,
                                                              int H, int W, int r) {
    extern __shared__ uint32_t lt[];  // [e][kCwPx + 2r]
    const int e = 2 * r + 1, tw = kCwPx + 2 * r, area = e * e;
    const int y = blockIdx.y, x0 = blockIdx.x * kCwPx;
    for (int q = threadIdx.x; q < e * tw; q += kCwT) {
        const int ty = q / tw, yy = y - r + ty, xx = x0 - r + q - ty * tw;
        uint32_t v = kCwOut;
        if (yy >= 0 && yy < H && xx >= 0 && xx < W) {
            const uint8_t *p = lab + 3 * ((size_t)yy * W + xx);
            v = (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16);
        }
        lt[q] = v;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int px = threadIdx.x >> 5; px < kCwPx; px += kCwT / 32) {
        const int x = x0 + px;
        if (x >= W) return;
        const uint32_t c = lt[r * tw + px + r];
        float *out = w + ((size_t)y * W + x) * area;
        int ky = lane / e, kx = lane - ky * e;
        const int sy = 32 / e, sx = 32 - sy * e;  // a step of 32 along the window
#pragma unroll 4
        for (int k = lane; k < area; k += 32) {
            const uint32_t q = lt[ky * tw + px + kx];
            const uint32_t ad = __vabsdiffu4(c, q);
            out[k] = q & kCwOut ? 0.f : __fmul_rn(__ldg(pw + k), __ldg(g + __dp4a(ad, ad, 0u)));
            ky += sy;
            kx += sx;
            if (kx >= e) {
                kx -= e;
                ky++;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Aggregation by weight arrays over tiles of 64 pixels x DC disparities, a thread on
// 4 x 4 entries.  L2R (seq/AdaptiveWeightAggregation.cpp:73-111) takes the weights of the
// pixels x and x - d; R2L (out of place, :113-150) those of the window pixel and of the
// window pixel + d.  A window row is added in pieces of at most kAmTaps taps, whatever the
// radius.  Per piece the block stages, by cp.async, the cost columns (wrapped), the
// reference weights wR[k][pixel] and the target weights wT[k][u], u = pixel -+ disparity,
// each read once (consecutive floats of a pixel) and turned so that a thread's weights are
// 16-byte loads; every entry then adds the piece's taps in order.  Padding entries take
// clamped or stale cells and are never written.
// Bound: the FP32 pipe (4 operations a tap and entry: 150 us of 327 us at 240x180, D = 32,
// 33x33) and the waits of a block for its next piece; the SM's other four blocks fill some
// of those (two buffers a block leave three blocks: 369 us; pieces of 17 taps read the
// cost columns more often: 440 us).  A thread per entry read both weights of every tap
// from 32 different lines: 2027 us.
constexpr int kAmTaps = 33;
constexpr int kAmTX = 64;
// row pitch of the turned target weights: 4 mod 32, so that consecutive taps of a pixel
// fall in banks 4 apart (odd strides would lose the 16-byte loads)
template <int DC> constexpr int kAmTP = (kAmTX + DC + 31) / 32 * 32 + 4;
// floats of one piece's buffer: cost columns, wR, wT
template <int DC> constexpr int kAmBuf = (kAmTX + kAmTaps - 1) * (DC + 4) + kAmTaps * (kAmTX + 4) + kAmTaps * kAmTP<DC>;

__device__ __forceinline__ void copy4(uint32_t dst, const float *src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <int DC, bool R2L>
__global__ void __launch_bounds__(4 * DC, DC == 64 ? 3 : 5)
    k_aw_tile(const float *__restrict__ wr, const float *__restrict__ wt, const float *__restrict__ cost,
              float *__restrict__ out, int H, int W, int D, int r, int vec_in, int vec_out, float zero) {
    constexpr int T = 4 * DC, NT = kAmTX + DC - 1, TP = kAmTP<DC>, RP = kAmTX + 4, CP = DC + 4, DG = DC / 4;
    const int e = 2 * r + 1, area = e * e;
    extern __shared__ __align__(16) float am[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dd0 = 4 * (tid % DG), px0 = 4 * (tid / DG);
    const int y = blockIdx.y, x0 = blockIdx.x * kAmTX, dc0 = blockIdx.z * DC;
    auto col = [&](int x) { return imin(imax(wrap1(x, W), 0), W - 1); };
    const float2 z2 = make_float2(zero, zero);
    float2 sw[4][2], sc[4][2];  // disparity pairs (dd0 + 2h, dd0 + 2h + 1) of pixel px0 + j
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) sw[j][h] = sc[j][h] = make_float2(0.f, 0.f);
    // a window row's e taps in pieces of kn (the last: the rest)
    const int pieces = (e + kAmTaps - 1) / kAmTaps, kn = (e + pieces - 1) / pieces, last = e - (pieces - 1) * kn;
    auto stage = [&](int dy, int piece) {
        const uint32_t cs = (uint32_t)__cvta_generic_to_shared(am), wrs = cs + 4 * (kAmTX + kAmTaps - 1) * CP,
                       wts = wrs + 4 * kAmTaps * RP;
        const int yy = wrap1(y + dy, H), kb = piece * kn, n = piece + 1 < pieces ? kn : last;
        const float *crow = cost + (size_t)yy * W * D;
        if (vec_in) {
            for (int q = tid; q < (kAmTX + n - 1) * DG; q += T) {
                const int xi = q / DG, dd = q % DG * 4;
                const bool in = dc0 + dd < D;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(cs + 4 * (xi * CP + dd)),
                             "l"(crow + (size_t)col(x0 - r + kb + xi) * D + (in ? dc0 + dd : 0)), "r"(in ? 16 : 0)
                             : "memory");
            }
        } else {
            for (int q = tid; q < (kAmTX + n - 1) * DC; q += T) {
                const int xi = q / DC, dd = q % DC;
                const bool in = dc0 + dd < D;
                copy4(cs + 4 * (xi * CP + dd), crow + (size_t)col(x0 - r + kb + xi) * D + (in ? dc0 + dd : 0), in ? 4 : 0);
            }
        }
        // weights of columns first .., in the pixel's own row (L2R) or the window's (R2L), taps
        // kb .. kb + n - 1: a warp per weight pixel, lane = tap, and tap 32 (33 x 33 windows)
        // a thread per pixel.  R2L: tap k of pixel x is window pixel q = x + k (from first),
        // so dst[k][q - k].
        auto turn = [&](const float *__restrict__ w, uint32_t dst, int pitch, int nu, int first) {
            const int np = R2L ? nu + n - 1 : nu;  // weight pixels
            const float *row = w + (size_t)(R2L ? yy : y) * W * area + (dy + r) * e + kb;
            if (lane < n) {
                const uint32_t o = dst + 4 * (lane * pitch - (R2L ? lane : 0));
#pragma unroll 4
                for (int q = warp; q < np; q += T / 32)
                    if (!R2L || (unsigned)(q - lane) < (unsigned)nu)
                        copy4(o + 4 * q, row + (size_t)col(first + q) * area + lane, 4);
            }
            if (n > 32)
                for (int q = tid; q < np; q += T)
                    if (!R2L || (unsigned)(q - 32) < (unsigned)nu)
                        copy4(dst + 4 * (32 * pitch + q - (R2L ? 32 : 0)), row + (size_t)col(first + q) * area + 32, 4);
        };
        turn(wr, wrs, RP, kAmTX, R2L ? x0 - r + kb : x0);
        turn(wt, wts, TP, NT, R2L ? x0 + dc0 - r + kb : x0 - dc0 - (DC - 1));
    };
    const float *Cs = am, *wRs = Cs + (kAmTX + kAmTaps - 1) * CP, *wTs = wRs + kAmTaps * RP;
    for (int t = 0; t < e * pieces; t++) {
        const int dy = t / pieces - r, piece = t - (dy + r) * pieces;
        const int n = piece + 1 < pieces ? kn : last;
        __syncthreads();  // the previous piece is consumed
        stage(dy, piece);
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        // target index of entry (j, i): px0 + j - dd0 - i + DC - 1 (L2R), px0 + j + dd0 + i (R2L)
        const float *wtp = wTs + (R2L ? px0 + dd0 : px0 - dd0 + DC - 4), *wrp = wRs + px0;
        const float *cp = Cs + px0 * CP + dd0;
        float4 win[4];  // cost columns kx .. kx + 3 of the thread's first pixel
#pragma unroll
        for (int q = 0; q < 3; q++) win[q] = *reinterpret_cast<const float4 *>(cp + q * CP);
        auto tap = [&](const float4 &c0, const float4 &c1, const float4 &c2, const float4 &c3) {
            const float4 a = *reinterpret_cast<const float4 *>(wrp);
            const float4 b0 = *reinterpret_cast<const float4 *>(wtp), b1 = *reinterpret_cast<const float4 *>(wtp + 4);
            const float wa[4] = {a.x, a.y, a.z, a.w};
            const float wb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            const float4 c[4] = {c0, c1, c2, c3};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float cj[4] = {c[j].x, c[j].y, c[j].z, c[j].w};
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    // C w by a packed multiply-add with a zero the compiler cannot see: it rounds
                    // like the multiply alone (a packed product feeding a packed add would be fused)
                    const float w0 = __fmul_rn(wa[j], wb[R2L ? j + 2 * h : j - 2 * h + 3]);
                    const float w1 = __fmul_rn(wa[j], wb[R2L ? j + 2 * h + 1 : j - 2 * h + 2]);
                    sw[j][h] = __fadd2_rn(sw[j][h], make_float2(w0, w1));
                    sc[j][h] = __fadd2_rn(sc[j][h], __ffma2_rn(make_float2(cj[2 * h], cj[2 * h + 1]), make_float2(w0, w1), z2));
                }
            }
            wrp += RP;
            wtp += TP;
        };
        int kx = 0;
        cp += 3 * CP;
        for (; kx + 4 <= n; kx += 4, cp += 4 * CP) {
            const float4 n0 = *reinterpret_cast<const float4 *>(cp), n1 = *reinterpret_cast<const float4 *>(cp + CP);
            const float4 n2 = *reinterpret_cast<const float4 *>(cp + 2 * CP);
            const float4 n3 = *reinterpret_cast<const float4 *>(cp + 3 * CP);
            tap(win[0], win[1], win[2], n0);
            tap(win[1], win[2], n0, n1);
            tap(win[2], n0, n1, n2);
            tap(n0, n1, n2, n3);
            win[0] = n1;
            win[1] = n2;
            win[2] = n3;
        }
        for (; kx < n; kx++, cp += CP) {
            const float4 n = *reinterpret_cast<const float4 *>(cp);
            tap(win[0], win[1], win[2], n);
            win[0] = win[1];
            win[1] = win[2];
            win[2] = n;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int x = x0 + px0 + j, d = dc0 + dd0;
        if (x >= W) break;
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            v[i] = __fdiv_rn(i & 1 ? sc[j][i >> 1].y : sc[j][i >> 1].x, i & 1 ? sw[j][i >> 1].y : sw[j][i >> 1].x);
        float *o = out + ((size_t)y * W + x) * D + d;
        if (vec_out) {
            if (d < D) *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (d + i < D) o[i] = v[i];
        }
    }
}

// A thread per entry, for ranges and windows that leave most of a tile idle (aw_tiles).  Its
// weights come from up to 32 different lines a tap.
// L2R: the weights of the pixels x and x - d.
__global__ void k_aw_entry_l2r(const float *__restrict__ wr, const float *__restrict__ wt,
                               const float *__restrict__ cost, float *__restrict__ out, int H, int W, int D, int r) {
    const int y = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * D) return;
    const int x = i / D, d = i - x * D;
    const int e = 2 * r + 1, area = e * e;
    const float *a = wr + ((size_t)y * W + x) * area;
    const float *b = wt + ((size_t)y * W + tar_col(x, d, W, 1)) * area;
    float sw = 0.f, sc = 0.f;
    int k = 0;
    for (int dy = -r; dy <= r; dy++) {
        const float *crow = cost + (size_t)wrap1(y + dy, H) * W * D + d;
        for (int dx = -r; dx <= r; dx++, k++) {
            const float wgt = __fmul_rn(a[k], b[k]);
            sw = __fadd_rn(sw, wgt);
            sc = __fadd_rn(sc, __fmul_rn(crow[(size_t)wrap1(x + dx, W) * D], wgt));
        }
    }
    out[((size_t)y * W + x) * D + d] = __fdiv_rn(sc, sw);
}
// R2L: those of the window pixel and of the window pixel + d.
__global__ void k_aw_entry_r2l(const float *__restrict__ wr, const float *__restrict__ wt,
                               const float *__restrict__ cost, float *__restrict__ out, int H, int W, int D, int r) {
    const int y = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * D) return;
    const int x = i / D, d = i - x * D;
    const int e = 2 * r + 1, area = e * e;
    float sw = 0.f, sc = 0.f;
    int k = 0;
    for (int dy = -r; dy <= r; dy++) {
        const size_t row = (size_t)wrap1(y + dy, H) * W;
        for (int dx = -r; dx <= r; dx++, k++) {
            const int xr = wrap1(x + dx, W), xt = wrap1(x + dx + d, W);
            const float wgt = __fmul_rn(wr[(row + xr) * area + k], wt[(row + xt) * area + k]);
            sw = __fadd_rn(sw, wgt);
            sc = __fadd_rn(sc, __fmul_rn(cost[(row + xr) * D + d], wgt));
        }
    }
    out[((size_t)y * W + x) * D + d] = __fdiv_rn(sc, sw);
}

// ---------------------------------------------------------------------------
static dim3 row_grid(long per_row, int H, int threads) { return dim3((unsigned)((per_row + threads - 1) / threads), H); }

void launch_compute_weights(cudaStream_t s, const uint8_t *lab, const float *pw, const float *g, float *w, int H, int W,
                            int r) {
    // the tile's 48 KB end at radius 51; windows below 32 weights would leave lanes of the tile's
    // warps without one (640x480: r = 1 17 us against 41, r = 2 37 and 45)
    if (r > 2 && cw_smem(r) <= 48 * 1024) {
        k_compute_weights_tile<<<dim3((W + kCwPx - 1) / kCwPx, H), kCwT, cw_smem(r), s>>>(lab, pw, g, w, H, W, r);
        return;
    }
    const long area = (long)(2 * r + 1) * (2 * r + 1);
    k_compute_weights<<<row_grid(W * area, H, 256), 256, 0, s>>>(lab, pw, g, w, H, W, r);
}

// 32 disparities a tile where that pads less than 64.  A thread per entry where the tiles'
// disparities are so many more than D that their share of idle lanes, and the waits of a
// tile for its few taps, cost more than the weights' lines: up to D = 64, below the lines
// D (24 + 10 r) = 24 * 32 and D (24 + 16 r) = 24 * 64, fitted to 640x480 and 240x180 (L2R, entry
// against tile: 640x480 r = 1, D = 20 91 and 105 us, D = 32 145 and 104, D = 33 148 and 197; r = 3,
// D = 12 203 and 236, D = 16 271 and 237; 240x180 r = 8, D = 4 80 and 122, D = 8 equal; r = 16,
// D = 4 278 and 330).  Images with fewer tiles than half the SMs: radii up to 6, and D below 32
// except for large L2R windows (64x48, r = 8, D = 16: L2R 37 and 42 us, R2L 43 and 84;
// L2R r = 16 124 and 105; these take tiles at D = 1 too, 240x180 437 and 376).
template <bool R2L>
static void aw_tiles(cudaStream_t s, const float *wr, const float *wt, const float *cost, float *out, int H, int W,
                     int D, int r) {
    const int dc = (D + 31) / 32 < 2 * ((D + 63) / 64) ? 32 : 64, padded = (D + dc - 1) / dc * dc;
    const long tiles = (long)((W + kAmTX - 1) / kAmTX) * H * (padded / dc);
    const bool few = 2 * tiles < sm_count();
    bool entry = D <= 64 && D * (24 + (dc == 32 ? 10 : 16) * r) < 24 * dc;
    if (few) entry = r <= 6 || (D < 32 && (R2L || r <= 8));
    if (!R2L && r > 8 && D == 1) entry = false;
    if (entry) {
        const auto kern = R2L ? k_aw_entry_r2l : k_aw_entry_l2r;
        kern<<<row_grid((long)W * D, H, 128), 128, 0, s>>>(wr, wt, cost, out, H, W, D, r);
        return;
    }
    auto go = [&](auto kern, int dc, int floats) {
        const size_t smem = (size_t)floats * sizeof(float);
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        // 16-byte copies of cost columns and results where each starts on 16 bytes
        const int vi = D % 4 == 0 && ((uintptr_t)cost & 15) == 0 ? 1 : 0, vo = D % 4 == 0 && ((uintptr_t)out & 15) == 0 ? 1 : 0;
        kern<<<dim3((W + kAmTX - 1) / kAmTX, H, (D + dc - 1) / dc), 4 * dc, smem, s>>>(wr, wt, cost, out, H, W, D, r,
                                                                                     vi, vo, 0.f);
    };
    if (dc == 32) go(k_aw_tile<32, R2L>, 32, kAmBuf<32>);
    else go(k_aw_tile<64, R2L>, 64, kAmBuf<64>);
}
void launch_aw_l2r_weights(cudaStream_t s, const float *wr, const float *wt, const float *cost, float *out, int H,
                           int W, int D, int r) {
    aw_tiles<false>(s, wr, wt, cost, out, H, W, D, r);
}
void launch_aw_r2l_weights(cudaStream_t s, const float *wr, const float *wt, const float *cost, float *out, int H,
                           int W, int D, int r) {
    aw_tiles<true>(s, wr, wt, cost, out, H, W, D, r);
}

}  // namespace rts
