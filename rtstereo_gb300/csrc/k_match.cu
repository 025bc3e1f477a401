// k_match.cu -- matching-cost kernels (module form of seq/PixelBasedCost.cpp,
// seq/CensusTransform.cpp, seq/RankFilter.cpp, seq/ConvolveImage.cpp,
// seq/NCCDisparity.cpp, seq/CombineCost.cpp).
//
// Float arithmetic that must match the reference bit for bit is written with
// explicit round-to-nearest intrinsics in the reference's order; the library
// is compiled with -fmad=false so no multiply-add is fused behind our back.
#include <algorithm>

#include "rts_common.cuh"

namespace rts {

// ---------------------------------------------------------------------------
// Cost volumes from two images: cost[y][x][d] = K::cost(ref word of x, target word of
// x -+ d).  Block per (row, kRowTX pixels): the words of the pixels and of every target
// column they meet (wrapped once, D <= W) are made once in shared memory, target column u
// in array u mod 4; a thread makes 4 consecutive disparities of a pixel, lanes on
// consecutive groups (so on consecutive words), and stores them as 16 bytes where every
// group starts on 16 (`vec`).  TX pixels a block: 32, and more where a pixel has few groups
// (128 up to D = 16, 256 up to D = 8), so that every thread has some.  magic = ceil(2^20 /
// groups): i / groups for i below 32 * 64 (the error i / 2^20 is below 1 / 64, at most
// 1 / groups; with 128 and 256 pixels i is below 512).
// Bound: instruction issue, then the volume's write (a division, two dependent image
// reads and byte loads per entry before: colour AD 640x480, D = 64 79 us; an entry a
// thread 30 us; 25 us now; gray AD 1280x720, D = 64 172, 67 and 57 us).
template <typename K, int kRowTX>
__global__ void __launch_bounds__(256) k_cost_rows(K k, float *__restrict__ cost, int D, int W, int dir, int vec,
                                                   uint32_t magic) {
    using T = typename K::T;
    constexpr int kRowNT = (kRowTX + (kRowTX == 32 ? 256 : kRowTX == 128 ? 16 : 8)) / 4;
    __shared__ T ref[kRowTX], tar[4][kRowNT];
    const int tid = threadIdx.x, x0 = blockIdx.x * kRowTX, ng = (D + 3) >> 2, Dp = 4 * ng;
    const size_t row = (size_t)blockIdx.y * W;
    // L2R: target column u of tar is x0 - Dp + u, entry (x, d) at u = x + Dp - d; R2L: x0 + u, x + d
    const int t0 = dir > 0 ? x0 - Dp : x0;
    for (int i = tid; i < kRowTX + Dp; i += 256) {
        int xt = t0 + i;
        if (xt < 0) xt += W;                                  // seq/PixelBasedCost.cpp:19-20
        else if (dir < 0 && xt >= W) xt -= W;                 // :32-33
        tar[i & 3][i >> 2] = k.load_tar(row + imax(imin(xt, W - 1), 0));  // columns of no pixel are clamped
    }
    if (tid < kRowTX) ref[tid] = k.load_ref(row + imin(x0 + tid, W - 1));
    __syncthreads();
    const int n = imin(kRowTX, W - x0) * ng;
    float *out = cost + (row + x0) * D;
#pragma unroll 2
    for (int i = tid; i < n; i += 256) {
        const int x = (int)(((uint32_t)i * magic) >> 20), d = 4 * (i - x * ng);
        const T a = ref[x];
        const int u = dir > 0 ? x + Dp - d : x + d;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int uj = dir > 0 ? u - j : u + j;
            v[j] = k.cost(a, tar[uj & 3][uj >> 2]);
        }
        float *o = out + (size_t)x * D + d;
        if (vec) {
            *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (d + j < D) o[j] = v[j];
        }
    }
}

// seq/PixelBasedCost.cpp:22 abs of an int difference
struct CostGray {
    using T = uint32_t;
    const uint8_t *r, *t;
    __device__ T load_ref(size_t p) const { return r[p]; }
    __device__ T load_tar(size_t p) const { return t[p]; }
    __device__ float cost(T a, T b) const { return (float)abs((int)a - (int)b); }
};
// seq/PixelBasedCost.cpp:48-50 float difference then sign flip
struct CostFloat {
    using T = float;
    const float *r, *t;
    __device__ T load_ref(size_t p) const { return r[p]; }
    __device__ T load_tar(size_t p) const { return t[p]; }
    __device__ float cost(T a, T b) const {
        const float v = __fsub_rn(a, b);
        return v < 0 ? -v : v;
    }
};
// seq/PixelBasedCost.cpp:86-91,106-112: min(sad, trunc), then (float)1/(float)3 * v
struct CostColor {
    using T = uint32_t;  // packed RGB
    const uint8_t *r, *t;
    int use_trunc, norm;
    float trunc;
    static __device__ T pack(const uint8_t *q) {
        return (uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16);
    }
    __device__ T load_ref(size_t p) const { return pack(r + 3 * p); }
    __device__ T load_tar(size_t p) const { return pack(t + 3 * p); }
    __device__ float cost(T a, T b) const {
        float v = (float)__vsadu4(a, b);
        if (use_trunc) v = (v > trunc) ? trunc : v;
        return norm ? __fmul_rn(1.0f / 3.0f, v) : v;
    }
};
// seq/CensusTransform.cpp:60, from packed codes of NW words
template <int NW> struct CostHamming {
    struct T {
        uint64_t w[NW];
    };
    const uint64_t *r, *t;
    static __device__ T load(const uint64_t *c, size_t p) {
        T v;
#pragma unroll
        for (int j = 0; j < NW; j++) v.w[j] = c[p * NW + j];
        return v;
    }
    __device__ T load_ref(size_t p) const { return load(r, p); }
    __device__ T load_tar(size_t p) const { return load(t, p); }
    __device__ float cost(const T &a, const T &b) const {
        int cnt = 0;
#pragma unroll
        for (int j = 0; j < NW; j++) cnt += __popcll(a.w[j] ^ b.w[j]);
        return (float)cnt;
    }
};

// ---------------------------------------------------------------------------
// Census.  Module form writes the reference's bool layout, one byte per bit;
// the pipeline uses packed 64-bit words (bit k of the window in word k/64).

// any window: a thread per bit
__global__ void k_census_bits(const uint8_t *__restrict__ img, uint8_t *__restrict__ bits, int hr, int wr, int H,
                              int W) {
    const int y = blockIdx.y;
    const int bw = 2 * wr + 1, nb = (2 * hr + 1) * bw;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * nb) return;
    const int x = i / nb, k = i - x * nb;
    const int dy = k / bw - hr, dx = k - (k / bw) * bw - wr;
    const uint8_t c = img[(size_t)y * W + x];
    const uint8_t n = img[(size_t)wrap1(y + dy, H) * W + wrap1(x + dx, W)];
    bits[((size_t)y * W + x) * nb + k] = (c > n) ? 1 : 0;  // seq/CensusTransform.cpp:31 strict
}

// Windows of up to kBitsMax bits: block per 128 consecutive pixels (of all rows), a
// thread per pixel.  The pixel's bytes go to shared memory, then the block's 128 nb
// bytes leave as 16-byte lines (`wide`: a 16-byte aligned output; 128 nb is a multiple
// of 16, so every block then starts on one).  Bound: the window's reads (one byte
// load and compare a bit; two divisions a bit before: 640x480, 9x7 72 us an image; 19 us
// now).
constexpr int kBitsT = 128, kBitsMax = 256;
template <bool WIN>  // the 9x7 window, unrolled
__global__ void __launch_bounds__(kBitsT) k_census_bits_px(const uint8_t *__restrict__ img, uint8_t *__restrict__ bits,
                                                           int hr_, int wr_, int H, int W, int wide) {
    extern __shared__ __align__(16) uint8_t sb[];  // [128][nb]
    const int hr = WIN ? 4 : hr_, wr = WIN ? 3 : wr_;
    const int nb = (2 * hr + 1) * (2 * wr + 1), tid = threadIdx.x;
    const long np = (long)H * W, p0 = (long)blockIdx.x * kBitsT, p = p0 + tid;
    if (p < np) {
        const int y = (int)(p / W), x = (int)(p - (long)y * W);
        const uint8_t c = img[p];
        uint8_t *o = sb + tid * nb;
        if (x >= wr && x < W - wr && y >= hr && y < H - hr) {
            // the window inside the image: no wrapping
            const uint8_t *row = img + p - (size_t)hr * W - wr;
            if constexpr (WIN) {
                int v[63];
#pragma unroll
                for (int k = 0; k < 63; k++) v[k] = row[(size_t)(k / 7) * W + k % 7];
#pragma unroll
                for (int k = 0; k < 63; k++) o[k] = (uint8_t)((uint32_t)(v[k] - c) >> 31);
            } else {
                for (int dy = -hr; dy <= hr; dy++, row += W)
                    for (int dx = 0; dx <= 2 * wr; dx++) *o++ = c > row[dx] ? 1 : 0;
            }
        } else {
            for (int dy = -hr; dy <= hr; dy++) {
                const uint8_t *row = img + (size_t)wrap1(y + dy, H) * W;
                for (int dx = -wr; dx <= wr; dx++) *o++ = c > row[wrap1(x + dx, W)] ? 1 : 0;
            }
        }
    }
    __syncthreads();
    const int n = (int)(np - p0 < kBitsT ? np - p0 : kBitsT) * nb;
    uint8_t *out = bits + (size_t)p0 * nb;
    int i = 0;
    if (wide) {
        for (int q = tid; q < n / 16; q += kBitsT)
            reinterpret_cast<uint4 *>(out)[q] = reinterpret_cast<const uint4 *>(sb)[q];
        i = n / 16 * 16;
    }
    for (i += tid; i < n; i += kBitsT) out[i] = sb[i];
}

template <int NW>
__global__ void k_census_codes(const uint8_t *__restrict__ img, uint64_t *__restrict__ codes, int hr, int wr,
                               int H, int W) {
    const int y = blockIdx.y;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= W) return;
    const uint8_t c = img[(size_t)y * W + x];
    uint64_t w[NW];
#pragma unroll
    for (int j = 0; j < NW; j++) w[j] = 0;
    int k = 0;
    if (NW == 1 && x >= wr && x < W - wr && y >= hr && y < H - hr) {
        // the window inside the image: no wrapping
        const uint8_t *row = img + (size_t)(y - hr) * W + x - wr;
        for (int dy = -hr; dy <= hr; dy++, row += W)
            for (int dx = 0; dx <= 2 * wr; dx++, k++) w[0] |= (uint64_t)(c > row[dx]) << k;
    } else {
        for (int dy = -hr; dy <= hr; dy++) {
            const uint8_t *row = img + (size_t)wrap1(y + dy, H) * W;
            for (int dx = -wr; dx <= wr; dx++, k++) {
                const uint64_t bit = (c > row[wrap1(x + dx, W)]) ? 1ull : 0ull;
#pragma unroll
                for (int j = 0; j < NW; j++)
                    if ((k >> 6) == j) w[j] |= bit << (k & 63);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NW; j++) codes[((size_t)y * W + x) * NW + j] = w[j];
}

// The bool layout packed again: block per 128 pixels, their 128 nb bytes staged in
// shared memory by 16-byte loads (`wide`: a 16-byte aligned input), then a thread per
// pixel (its own bytes straight from memory are 32 different lines a load; packing and
// distances 640x480, D = 64: 88 us before, 54 us now).
template <int NW>
__global__ void __launch_bounds__(kBitsT) k_bits_pack(const uint8_t *__restrict__ bits, uint64_t *__restrict__ codes,
                                                      int nb, long npix, int wide) {
    extern __shared__ __align__(16) uint8_t sb[];  // [128][nb]
    const int tid = threadIdx.x;
    const long p0 = (long)blockIdx.x * kBitsT;
    const int np = (int)(npix - p0 < kBitsT ? npix - p0 : kBitsT), n = np * nb;
    const uint8_t *in = bits + (size_t)p0 * nb;
    int i = 0;
    if (wide) {
        for (int q = tid; q < n / 16; q += kBitsT)
            reinterpret_cast<uint4 *>(sb)[q] = reinterpret_cast<const uint4 *>(in)[q];
        i = n / 16 * 16;
    }
    for (i += tid; i < n; i += kBitsT) sb[i] = in[i];
    __syncthreads();
    if (tid >= np) return;
    const uint8_t *b = sb + tid * nb;
#pragma unroll
    for (int j = 0; j < NW; j++) {
        uint64_t w = 0;
        const int e = imin(64, nb - 64 * j);
#pragma unroll 8
        for (int k = 0; k < e; k++) w |= (uint64_t)(b[64 * j + k] != 0) << k;
        codes[(size_t)(p0 + tid) * NW + j] = w;
    }
}

// ---------------------------------------------------------------------------
// Window filters of an image: rank, LoG convolution, window mean.  Block per 64 x 16
// pixels (64 x 4 in small images); their wrapped border is staged in shared memory once
// (single wrap: radii are below the image's sides), a thread makes four (one) pixels of a column.  A window of up to
// kWinMax pixels of border takes them; WR, WC: the radii as constants (the usual windows,
// loops unrolled) or -1.  Bound: the window's shared-memory reads and operations
// (1280x720: rank 7x7 33 us, LoG 5x5 21 us an image when every window pixel was a
// wrapped read of the image; 14 and 13 us now).
constexpr int kWinTX = 64, kWinT = 256, kWinMax = 64;

template <typename F, int WR, int WC, int kWinTY>
__global__ void __launch_bounds__(kWinT) k_window(const uint8_t *__restrict__ img, typename F::Out *__restrict__ out,
                                                  F f, int H, int W, int hr_, int wr_) {
    extern __shared__ uint8_t wt[];  // [16 + 2 hr][64 + 2 wr]
    const int hr = WR >= 0 ? WR : hr_, wr = WC >= 0 ? WC : wr_;
    const int tw = kWinTX + 2 * wr, th = kWinTY + 2 * hr, x0 = blockIdx.x * kWinTX, y0 = blockIdx.y * kWinTY;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = warp; r < th; r += kWinT / 32) {
        // rows and columns past the last pixel's window are clamped into range (never used)
        const uint8_t *row = img + (size_t)wrap1(imin(y0 - hr + r, H - 1 + hr), H) * W;
        uint8_t g[6];  // the row's (at most 64 + 2 kWinMax) columns in flight together
#pragma unroll
        for (int k = 0; k < 6; k++) {
            const int c = lane + 32 * k;
            g[k] = c < tw ? row[wrap1(imin(x0 - wr + c, W - 1 + wr), W)] : (uint8_t)0;
        }
#pragma unroll
        for (int k = 0; k < 6; k++)
            if (lane + 32 * k < tw) wt[r * tw + lane + 32 * k] = g[k];
    }
    __syncthreads();
    const int px = threadIdx.x & (kWinTX - 1), x = x0 + px;
    if (x >= W) return;
#pragma unroll
    for (int i = 0; i < kWinTY; i += kWinT / kWinTX) {
        const int py = i + threadIdx.x / kWinTX, y = y0 + py;
        if (y >= H) return;
        const uint8_t *w = wt + py * tw + px;  // the window's first pixel
        typename F::Acc acc = f.begin(w[hr * tw + wr]);
        if constexpr (WR >= 0) {
#pragma unroll
            for (int dy = 0; dy <= 2 * WR; dy++)
#pragma unroll
                for (int dx = 0; dx <= 2 * WC; dx++) f.add(acc, w[dy * tw + dx], dy * (2 * WC + 1) + dx);
        } else {
            for (int dy = 0, k = 0; dy <= 2 * hr; dy++)
                for (int dx = 0; dx <= 2 * wr; dx++, k++) f.add(acc, w[dy * tw + dx], k);
        }
        out[(size_t)y * W + x] = f.end(acc);
    }
}

// Rank transform (seq/RankFilter.cpp:11-35): 1 + #{q : I(q) < I(p)}, u8 wrap.
struct RankWin {
    using Out = uint8_t;
    struct Acc {
        int c, n;
    };
    __device__ Acc begin(int c) const { return Acc{c, 1}; }
    __device__ void add(Acc &a, int v, int) const { a.n += (uint32_t)(v - a.c) >> 31; }
    __device__ Out end(const Acc &a) const { return (uint8_t)a.n; }
};
// LoG convolution (seq/ConvolveImage.cpp:11-35): raster-order sum of rounded
// products, |.|, min 255.
struct ConvWin {
    using Out = float;
    using Acc = float;
    const float *mask;
    __device__ Acc begin(int) const { return 0.f; }
    __device__ void add(Acc &a, int v, int k) const { a = __fadd_rn(a, __fmul_rn((float)v, __ldg(mask + k))); }
    __device__ Out end(Acc a) const {
        a = (a > 0.f) ? a : -a;
        return (a > 255.f) ? 255.f : a;
    }
};
// Window mean for NCC (seq/NCCDisparity.cpp:24-35): raster-order float sum / area.  A: int
// where the sum stays below 2^24 (the float sums are then exact), else float.  The target
// mean of (x, d) equals this mean at column x-d (wrapped): the same pixels.
template <typename A> struct MeanWin {
    using Out = float;
    using Acc = A;
    float area;
    __device__ Acc begin(int) const { return 0; }
    __device__ void add(Acc &a, int v, int) const { a = a + (A)v; }
    __device__ Out end(Acc a) const { return __fdiv_rn((float)a, area); }
};

// windows whose border does not fit the tile (radius above kWinMax): a thread per pixel
template <typename F>
__global__ void k_window_any(const uint8_t *__restrict__ img, typename F::Out *__restrict__ out, F f, int H, int W,
                             int hr, int wr) {
    const int y = blockIdx.y;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= W) return;
    typename F::Acc acc = f.begin(img[(size_t)y * W + x]);
    int k = 0;
    for (int dy = -hr; dy <= hr; dy++) {
        const uint8_t *row = img + (size_t)wrap1(y + dy, H) * W;
        for (int dx = -wr; dx <= wr; dx++, k++) f.add(acc, row[wrap1(x + dx, W)], k);
    }
    out[(size_t)y * W + x] = f.end(acc);
}

// NCC (seq/NCCDisparity.cpp:50-71): nom = sum rv*tv, den = sqrtf(sum ((rv*rv)*tv)*tv)
// in tap (raster) order, the cell written only when den != 0.  Over tiles: block per (row y, 64 pixels,
// 64 disparities), each thread 4 pixels x 4 disparities.  Per chunk of taps the
// block stages, in tap (raster) order, {rv, rv*rv} of its 64 reference pixels and
// tv of the 127 target columns t = x - d it meets (rv = I - mean, tv likewise,
// seq/NCCDisparity.cpp:55-62).  An entry's (nom, den) pair then takes per tap
//   rv*tv, ((rv*rv)*tv)*tv as scalar products, (nom, den) += (rv*tv, den term)
//   (one packed add)
// which are the reference's operations in its order.  A thread's 16 entries read
// 8 reference and 8 target floats per tap: four 16-byte shared loads, the
// target values held once (a {tv, tv} pair for a packed multiply would double
// the shared-memory traffic).  Bound: the FP32 pipe (5 operations a tap and entry), and the
// staging's latency: three blocks an SM (80 registers) rather than two (124) 1334 -> 1106 us
// for the two views of 1280x720, D = 64, 7x7; blocks whose windows do not wrap stage by one
// offset a tap (1468 us with the wraps, a volume cleared first and costs stored four
// bytes at a time).
constexpr int kNccTX = 64, kNccTD = 64, kNccTaps = 49;
static_assert(sizeof(float2) * kNccTaps * kNccTX + sizeof(float) * kNccTaps * (kNccTX + kNccTD) <= kSmemOptin,
              "NCC tile exceeds the shared-memory opt-in");
__global__ void __launch_bounds__(256, 3) k_ncc_tiled(const uint8_t *__restrict__ ref, const uint8_t *__restrict__ tar,
                                                   const float *__restrict__ mref, const float *__restrict__ mtar,
                                                   float *__restrict__ cost, int D, int H, int W, int hr, int wr,
                                                   int fill, int vec) {
    constexpr int NT = kNccTX + kNccTD - 1;       // target columns of a tile
    extern __shared__ __align__(16) unsigned char nsm[];
    float2 (*rq)[kNccTX] = reinterpret_cast<float2 (*)[kNccTX]>(nsm);                         // {rv, rv*rv}
    float (*tq)[NT + 1] = reinterpret_cast<float (*)[NT + 1]>(nsm + sizeof(float2) * kNccTaps * kNccTX);  // tv
    const int tid = threadIdx.x;
    // a warp's 16 disparity groups store one pixel's 64 costs as whole lines
    const int px0 = 4 * (tid >> 4), d0 = 4 * (tid & 15);
    const int y = blockIdx.y, x0 = blockIdx.x * kNccTX, dc0 = blockIdx.z * kNccTD;
    const int tbase = x0 - dc0 - (kNccTD - 1);    // target column of u = 0 (before wrapping)
    const int ew = 2 * wr + 1, taps = (2 * hr + 1) * ew;
    // the tap offsets {dy, dx} of a chunk, made once per chunk, and as one offset where no
    // window of the block wraps
    __shared__ int2 tapoff[kNccTaps];
    __shared__ int tapadd[kNccTaps];
    const bool inside = y >= hr && y + hr < H && tbase >= wr && x0 + kNccTX + wr <= W;
    float2 acc[4][4];  // (nom, den) of pixel px0 + j, disparity d0 + i
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[j][i] = make_float2(0.f, 0.f);
    for (int k0 = 0; k0 < taps; k0 += kNccTaps) {
        const int nk = min(kNccTaps, taps - k0);
        __syncthreads();  // the previous chunk is consumed
        if (tid < nk) {
            const int kk = k0 + tid, ry = kk / ew;
            tapoff[tid] = make_int2(ry - hr, kk - ry * ew - wr);
            tapadd[tid] = (ry - hr) * W + kk - ry * ew - wr;
        }
        __syncthreads();
        if (inside) {
            // reference and target cells as below, without the wraps
            const size_t row = (size_t)y * W;
            const int px = tid & (kNccTX - 1);
            const uint8_t *rp = ref + row + x0 + px;
            const float mr = mref[row + x0 + px];
#pragma unroll 4
            for (int k = tid >> 6; k < nk; k += 256 / kNccTX) {
                const float rv = __fsub_rn((float)rp[tapadd[k]], mr);
                rq[k][px] = make_float2(rv, __fmul_rn(rv, rv));
            }
            if (tid < 2 * NT) {
                const int u = tid < NT ? tid : tid - NT;
                const uint8_t *tp = tar + row + tbase + u;
                const float mt = mtar[row + tbase + u];
#pragma unroll 8
                for (int k = tid < NT ? 0 : 1; k < nk; k += 2) tq[k][u] = __fsub_rn((float)tp[tapadd[k]], mt);
            }
        } else {
            // reference cells: a thread keeps one pixel (its mean loaded once) over every
            // 4th tap of the chunk
            const int px = tid & (kNccTX - 1);
            const int x = min(x0 + px, W - 1);
            const float mr = mref[(size_t)y * W + x];
            for (int k = tid >> 6; k < nk; k += 256 / kNccTX) {
                const int2 to = tapoff[k];
                const float rv = __fsub_rn((float)ref[(size_t)wrap1(y + to.x, H) * W + wrap1(x + to.y, W)], mr);
                rq[k][px] = make_float2(rv, __fmul_rn(rv, rv));
            }
        }
        if (!inside && tid < 2 * NT) {
            // target cells: threads 0 .. 2 NT - 1 keep one column each over every other tap
            const int u = tid < NT ? tid : tid - NT;
            // t in [-W, 2W) for real entries; columns of padding entries clamped into range
            const int t = wrap1(max(min(tbase + u, W - 1), -W + 1), W);
            const float mt = mtar[(size_t)y * W + t];  // seq/NCCDisparity.cpp:37-48, same columns
            for (int k = tid < NT ? 0 : 1; k < nk; k += 2) {
                const int2 to = tapoff[k];
                const float tv = __fsub_rn((float)tar[(size_t)wrap1(y + to.x, H) * W + wrap1(t + to.y, W)], mt);
                tq[k][u] = tv;
            }
        }
        __syncthreads();
        // u index of (j, i): px0 + j - d0 - i + 63
        const int ub = px0 - d0 + kNccTD - 4;
#pragma unroll 7
        for (int k = 0; k < nk; k++) {
            float2 r[4];
            float tt[8];
            const float4 ra = *reinterpret_cast<const float4 *>(&rq[k][px0]);
            const float4 rb = *reinterpret_cast<const float4 *>(&rq[k][px0 + 2]);
            r[0] = make_float2(ra.x, ra.y); r[1] = make_float2(ra.z, ra.w);
            r[2] = make_float2(rb.x, rb.y); r[3] = make_float2(rb.z, rb.w);
            const float4 ta = *reinterpret_cast<const float4 *>(&tq[k][ub]);
            const float4 tb = *reinterpret_cast<const float4 *>(&tq[k][ub + 4]);
            tt[0] = ta.x; tt[1] = ta.y; tt[2] = ta.z; tt[3] = ta.w;
            tt[4] = tb.x; tt[5] = tb.y; tt[6] = tb.z; tt[7] = tb.w;
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    // scalar IEEE products (a product feeding a packed add stays unfused), the
                    // pair (rv*tv, ((rv*rv)*tv)*tv) added by one packed add
                    const float tv = tt[j - i + 3];
                    const float nt = __fmul_rn(r[j].x, tv);
                    const float dt = __fmul_rn(__fmul_rn(r[j].y, tv), tv);
                    acc[j][i] = __fadd2_rn(acc[j][i], make_float2(nt, dt));
                }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int x = x0 + px0 + j, d = dc0 + d0;
        if (x >= W || d >= D) break;
        float *o = cost + ((size_t)y * W + x) * D + d;
        float v[4];
        bool write[4], all = true;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            // a zero denominator leaves the cell unwritten (fill: writes 0)
            const float den = __fsqrt_rn(acc[j][i].y);  // seq/NCCDisparity.cpp:69
            v[i] = den != 0.f ? __fdiv_rn(acc[j][i].x, den) : 0.f;
            write[i] = den != 0.f || fill;
            all = all && write[i];
        }
        if (vec && all) {
            *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (d + i < D && write[i]) o[i] = v[i];
        }
    }
}

// LoG differences combined with census Hamming distances in one pass (composed:
// two volumes and k_combine, seq/Main.cpp:180-234 with LoG first and census
// second): the same expressions in the same order, one write of the volume.  A warp
// takes kLcPx consecutive pixels, lane = disparity.
constexpr int kLcPx = 8;

template <int NW>
__global__ void __launch_bounds__(256) k_cost_log_census(const float *__restrict__ lr, const float *__restrict__ lt,
                                                        const uint64_t *__restrict__ cr, const uint64_t *__restrict__ ct,
                                                        float *__restrict__ vol, int H, int W, int D,
                                                        const float *__restrict__ lut1, const float *__restrict__ lut2,
                                                        float lambda1, float lambda2) {
    const int y = blockIdx.y, lane = threadIdx.x & 31;
    const int xw = (blockIdx.x * 8 + (threadIdx.x >> 5)) * kLcPx;
    const size_t row = (size_t)y * W;
#pragma unroll 2
    for (int i = 0; i < kLcPx; i++) {
        const int x = xw + i;
        if (x >= W) return;
        const float a = lr[row + x];
        uint64_t ca[NW];
#pragma unroll
        for (int j = 0; j < NW; j++) ca[j] = cr[(row + x) * NW + j];
        float *out = vol + (row + x) * D;
        for (int d = lane; d < D; d += 32) {
            const int xt = x - d < 0 ? x - d + W : x - d;  // seq/PixelBasedCost.cpp:19-20
            float v1 = __fsub_rn(a, lt[row + xt]);         // seq/PixelBasedCost.cpp:48-50
            if (v1 < 0) v1 = -v1;
            int cnt = 0;
#pragma unroll
            for (int j = 0; j < NW; j++) cnt += __popcll(ca[j] ^ ct[(row + xt) * NW + j]);  // seq/CensusTransform.cpp:60
            out[d] = __fadd_rn(combine_term(v1, lut1, lambda1), combine_term((float)cnt, lut2, lambda2));
        }
    }
}

// In place, four entries a thread where both volumes are 16-byte aligned (n4 groups of
// four, then the rest one by one).  Bound: memory (two reads and a write), and for costs
// that are not whole numbers the expf and division of both terms (640x480, D = 64 whole
// numbers 79 -> 48 us; 1280x720, D = 64 others 237 -> 140 us).
__global__ void __launch_bounds__(256) k_combine(float *__restrict__ c1, const float *__restrict__ c2, long n, long n4,
                                                 const float *__restrict__ lut1, const float *__restrict__ lut2,
                                                 float lambda1, float lambda2) {
    const long step = (long)gridDim.x * 256, i0 = (long)blockIdx.x * 256 + threadIdx.x;
    auto one = [&](float a, float b) {
        return __fadd_rn(combine_term(a, lut1, lambda1), combine_term(b, lut2, lambda2));
    };
    for (long i = i0; i < n4; i += step) {
        float4 a = reinterpret_cast<float4 *>(c1)[i];
        const float4 b = reinterpret_cast<const float4 *>(c2)[i];
        a.x = one(a.x, b.x);
        a.y = one(a.y, b.y);
        a.z = one(a.z, b.z);
        a.w = one(a.w, b.w);
        reinterpret_cast<float4 *>(c1)[i] = a;
    }
    for (long i = 4 * n4 + i0; i < n; i += step) c1[i] = one(c1[i], c2[i]);
}

// ---------------------------------------------------------------------------
// launchers

static dim3 row_grid(long per_row, int H, int threads) { return dim3((unsigned)((per_row + threads - 1) / threads), H); }

template <typename K> static void cost_rows(cudaStream_t s, const K &k, float *cost, int D, int H, int W, int dir) {
    const int ng = (D + 3) / 4, vec = D % 4 == 0 && ((uintptr_t)cost & 15) == 0 ? 1 : 0;
    auto go = [&](auto kern, int tx) {
        kern<<<dim3((W + tx - 1) / tx, H), 256, 0, s>>>(k, cost, D, W, dir, vec, ((1u << 20) + ng - 1) / ng);
    };
    if (D <= 8) go(k_cost_rows<K, 256>, 256);
    else if (D <= 16) go(k_cost_rows<K, 128>, 128);
    else go(k_cost_rows<K, 32>, 32);
}
void launch_ad_gray(cudaStream_t s, const uint8_t *ref, const uint8_t *tar, float *cost, int D, int H, int W, int dir) {
    cost_rows(s, CostGray{ref, tar}, cost, D, H, W, dir);
}
void launch_ad_float(cudaStream_t s, const float *ref, const float *tar, float *cost, int D, int H, int W, int dir) {
    cost_rows(s, CostFloat{ref, tar}, cost, D, H, W, dir);
}
void launch_ad_color(cudaStream_t s, const uint8_t *ref, const uint8_t *tar, float *cost, int D, int H, int W, int dir,
                     int use_trunc, float trunc, int norm) {
    cost_rows(s, CostColor{ref, tar, use_trunc, norm, trunc}, cost, D, H, W, dir);
}
void launch_census_bits(cudaStream_t s, const uint8_t *img, uint8_t *bits, int hr, int wr, int H, int W) {
    const long nb = (long)(2 * hr + 1) * (2 * wr + 1);
    if (nb <= kBitsMax) {
        const int wide = ((uintptr_t)bits & 15) == 0 ? 1 : 0;
        const unsigned g = (unsigned)(((long)H * W + kBitsT - 1) / kBitsT);
        const size_t smem = (size_t)kBitsT * nb;
        if (hr == 4 && wr == 3) k_census_bits_px<true><<<g, kBitsT, smem, s>>>(img, bits, hr, wr, H, W, wide);
        else k_census_bits_px<false><<<g, kBitsT, smem, s>>>(img, bits, hr, wr, H, W, wide);
        return;
    }
    k_census_bits<<<row_grid(W * nb, H, 256), 256, 0, s>>>(img, bits, hr, wr, H, W);
}
int census_words(int hr, int wr) {
    const int nb = (2 * hr + 1) * (2 * wr + 1);
    return nb <= 64 ? 1 : nb <= 128 ? 2 : nb <= 256 ? 4 : 0;
}
void launch_census_codes(cudaStream_t s, const uint8_t *img, uint64_t *codes, int hr, int wr, int H, int W) {
    const dim3 g = row_grid(W, H, 128);
    switch (census_words(hr, wr)) {
    case 1: k_census_codes<1><<<g, 128, 0, s>>>(img, codes, hr, wr, H, W); break;
    case 2: k_census_codes<2><<<g, 128, 0, s>>>(img, codes, hr, wr, H, W); break;
    case 4: k_census_codes<4><<<g, 128, 0, s>>>(img, codes, hr, wr, H, W); break;
    }
}
void launch_bits_pack(cudaStream_t s, const uint8_t *bits, uint64_t *codes, int nb, long npix) {
    const unsigned g = (unsigned)((npix + kBitsT - 1) / kBitsT);
    const size_t smem = (size_t)kBitsT * nb;  // at most 32 KB
    const int wide = ((uintptr_t)bits & 15) == 0 ? 1 : 0;
    if (nb <= 64) k_bits_pack<1><<<g, kBitsT, smem, s>>>(bits, codes, nb, npix, wide);
    else if (nb <= 128) k_bits_pack<2><<<g, kBitsT, smem, s>>>(bits, codes, nb, npix, wide);
    else k_bits_pack<4><<<g, kBitsT, smem, s>>>(bits, codes, nb, npix, wide);
}
void launch_hamming(cudaStream_t s, const uint64_t *cr, const uint64_t *ct, float *cost, int nw, int D, int H, int W) {
    if (nw == 1) cost_rows(s, CostHamming<1>{cr, ct}, cost, D, H, W, 1);
    else if (nw == 2) cost_rows(s, CostHamming<2>{cr, ct}, cost, D, H, W, 1);
    else cost_rows(s, CostHamming<4>{cr, ct}, cost, D, H, W, 1);
}
template <typename F>
static void window(cudaStream_t s, const uint8_t *img, typename F::Out *out, const F &f, int H, int W, int hr, int wr) {
    if (hr > kWinMax || wr > kWinMax) {
        k_window_any<<<row_grid(W, H, 128), 128, 0, s>>>(img, out, f, H, W, hr, wr);
        return;
    }
    auto go = [&](auto kern, int ty) {
        kern<<<dim3((W + kWinTX - 1) / kWinTX, (H + ty - 1) / ty), kWinT,
               (size_t)(ty + 2 * hr) * (kWinTX + 2 * wr), s>>>(img, out, f, H, W, hr, wr);
    };
    // tiles of 4 rows where those of 16 are fewer than the SMs
    const bool few = (long)((W + kWinTX - 1) / kWinTX) * ((H + 15) / 16) < sm_count();
    if (few && hr == 2 && wr == 2) go(k_window<F, 2, 2, 4>, 4);
    else if (few && hr == 3 && wr == 3) go(k_window<F, 3, 3, 4>, 4);
    else if (few) go(k_window<F, -1, -1, 4>, 4);
    else if (hr == 2 && wr == 2) go(k_window<F, 2, 2, 16>, 16);
    else if (hr == 3 && wr == 3) go(k_window<F, 3, 3, 16>, 16);
    else go(k_window<F, -1, -1, 16>, 16);
}
void launch_rank(cudaStream_t s, const uint8_t *img, uint8_t *out, int m, int H, int W) {
    window(s, img, out, RankWin{}, H, W, m, m);
}
void launch_convolve(cudaStream_t s, const uint8_t *img, float *out, const float *mask, int H, int W, int hr, int wr) {
    window(s, img, out, ConvWin{mask}, H, W, hr, wr);
}
void launch_window_mean(cudaStream_t s, const uint8_t *img, float *mean, int H, int W, int hr, int wr) {
    const long area = (long)(2 * hr + 1) * (2 * wr + 1);
    if (255 * area < (1L << 24)) window(s, img, mean, MeanWin<int>{(float)area}, H, W, hr, wr);
    else window(s, img, mean, MeanWin<float>{(float)area}, H, W, hr, wr);
}
void launch_ncc(cudaStream_t s, const uint8_t *ref, const uint8_t *tar, const float *mref, const float *mtar,
                float *cost, int D, int H, int W, int hr, int wr, int fill) {
    const dim3 g((W + kNccTX - 1) / kNccTX, H, (D + kNccTD - 1) / kNccTD);
    const size_t smem = sizeof(float2) * kNccTaps * kNccTX + sizeof(float) * kNccTaps * (kNccTX + kNccTD);
    cudaFuncSetAttribute(k_ncc_tiled, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int vec = D % 4 == 0 && ((uintptr_t)cost & 15) == 0 ? 1 : 0;
    k_ncc_tiled<<<g, 256, smem, s>>>(ref, tar, mref, mtar, cost, D, H, W, hr, wr, fill, vec);
}
void launch_cost_log_census(cudaStream_t s, const float *lr, const float *lt, const uint64_t *cr, const uint64_t *ct,
                            int nw, float *vol, int D, int H, int W, const float *lut1, const float *lut2,
                            float lambda1, float lambda2) {
    const dim3 g((unsigned)((W + 8 * kLcPx - 1) / (8 * kLcPx)), H);
    if (nw == 1) k_cost_log_census<1><<<g, 256, 0, s>>>(lr, lt, cr, ct, vol, H, W, D, lut1, lut2, lambda1, lambda2);
    else if (nw == 2) k_cost_log_census<2><<<g, 256, 0, s>>>(lr, lt, cr, ct, vol, H, W, D, lut1, lut2, lambda1, lambda2);
    else k_cost_log_census<4><<<g, 256, 0, s>>>(lr, lt, cr, ct, vol, H, W, D, lut1, lut2, lambda1, lambda2);
}
void launch_combine(cudaStream_t s, float *c1, const float *c2, long n, const float *lut1, const float *lut2,
                    float lambda1, float lambda2) {
    const long n4 = (((uintptr_t)c1 | (uintptr_t)c2) & 15) == 0 ? n / 4 : 0;
    const long blocks = std::min((std::max(n4, n - 4 * n4) + 255) / 256, 152L * 64);
    k_combine<<<(unsigned)blocks, 256, 0, s>>>(c1, c2, n, n4, lut1, lut2, lambda1, lambda2);
}

}  // namespace rts
