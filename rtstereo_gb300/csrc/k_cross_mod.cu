// k_cross_mod.cu -- cross-based aggregation, module form
// (seq/CrossBasedAggregation.cpp:117-169).
//
// Per entry the reference's arithmetic in its order: the running sum along x, the
// row segment P[x + r] - P[x - l - 1], the segments' sum over the vertical arm top
// to bottom, the quotient by the pixel count.
#include <algorithm>

#include "rts_common.cuh"
#include "rts_vert_ring.h"

namespace rts {

// ---------------------------------------------------------------------------
// In-place running sum along x per (y, d) (seq/CrossBasedAggregation.cpp:117-125): one
// thread per chain, consecutive threads on consecutive d (coalesced).  Bound: memory
// latency, since a chain is serial and the H D chains are few.  So a thread loads the
// next kPreB columns before it adds and stores the current ones (as one load a step,
// each behind the previous column's store, 640x480, D = 64 took 282 us; 28 us now).
constexpr int kPreB = 32;
__global__ void __launch_bounds__(64) k_prefix_h(float *__restrict__ cost, int H, int W, int D) {
    const long i = (long)blockIdx.x * 64 + threadIdx.x;
    if (i >= (long)H * D) return;
    const int y = (int)(i / D), d = (int)(i - (long)y * D);
    float *p = cost + (size_t)y * W * D + d;
    float next[kPreB];
    auto load = [&](const float *q, int n) {
#pragma unroll
        for (int k = 0; k < kPreB; k++)
            if (k < n) next[k] = q[(size_t)k * D];
    };
    load(p, W);
    float acc = 0.f;
    for (int x = 0; x < W; x += kPreB, p += (size_t)kPreB * D) {
        float cur[kPreB];
#pragma unroll
        for (int k = 0; k < kPreB; k++) cur[k] = next[k];
        load(p + (size_t)kPreB * D, W - x - kPreB);
#pragma unroll
        for (int k = 0; k < kPreB; k++) {
            if (x + k >= W) break;
            acc = x + k == 0 ? cur[0] : __fadd_rn(cur[k], acc);  // column 0 stays as it is
            p[(size_t)k * D] = acc;
        }
    }
}

void launch_prefix_h(cudaStream_t s, float *cost, int H, int W, int D) {
    const long n = (long)H * D;
    k_prefix_h<<<(unsigned)((n + 63) / 64), 64, 0, s>>>(cost, H, W, D);
}

// ---------------------------------------------------------------------------
// Cross-based aggregation of a volume of running sums.  Arms made by findCross with
// lengths up to kModArm (the reference's are 17) take three kernels:
//   k_cross_pack  packs the four arm arrays into words (8 bytes a pixel and image) and
//                 raises *general where an arm is longer, negative or leaves the image
//   k_cross_seg   the row segment of every entry, once (an entry used to difference two
//                 running sums for every row of every cross it lies in)
//   k_cross_vol   vertical sums and quotients, each entry read once
// Any other arms (*general != 0, known on the device alone) take k_cross_aggr, which
// reads them as they are; each side returns at once where the other's case holds.
// 640x480, D = 64, arms near 17: k_cross_aggr alone 1348 us, the three kernels 192 us.
// So do volumes below kModSmall entries and ranges of one or two, where the launches cost more
// than they save (160x120, D = 16: 15 us of short arms and 27 of long ones, against 28 and 30).
constexpr size_t kModSmall = 512 * 1024;
constexpr int kModArm = 20;  // ring depth 48: 48 KB a block of 4 warps, 4 blocks an SM

__global__ void k_cross_pack(const int *__restrict__ hr, const int *__restrict__ ht, const int *__restrict__ vr,
                             const int *__restrict__ vt, uint2 *__restrict__ ra, uint2 *__restrict__ ta,
                             int *__restrict__ general, int H, int W) {
    const int y = blockIdx.y, x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= W) return;
    const size_t p = (size_t)y * W + x;
    const int l = hr[2 * p], r = hr[2 * p + 1], t = vr[2 * p], b = vr[2 * p + 1];
    const int tl = ht[2 * p], tr = ht[2 * p + 1], tt = vt[2 * p], tb = vt[2 * p + 1];
    // an entry's arms are minima with the reference's, so those alone bound them
    if (imin(imin(l, r), imin(t, b)) < 0 || imin(imin(tl, tr), imin(tt, tb)) < 0 ||
        imax(imax(l, r), imax(t, b)) > kModArm || l > x || r > W - 1 - x || t > y || b > H - 1 - y)
        *general = 1;
    auto word = [](int lo, int hi) { return (uint32_t)(imin(lo, 255) & 0xff) | ((uint32_t)(imin(hi, 255) & 0xff) << 16); };
    ra[p] = make_uint2(word(l, t), word(r, b));
    ta[p] = make_uint2(word(tl, tt), word(tr, tb));
}

// Row segments: block per (row, 32 pixels), a thread on every 256th entry of the
// block's 32 D.  magic = ceil(2^20 / D): i / D for i < 32 * 256 (the error i / 2^20 is
// below 1 / 256 <= 1 / D for i < 4096; the block's upper half starts at pixel 16).
constexpr int kSegTX = 32;
__global__ void __launch_bounds__(256) k_cross_seg(const float *__restrict__ pre, const uint2 *__restrict__ ra,
                                                   const uint2 *__restrict__ ta, float *__restrict__ seg,
                                                   const int *__restrict__ general, int W, int D, uint32_t magic) {
    __shared__ uint32_t ref[kSegTX], tar[kSegTX + 255];  // {l | r << 16}
    if (*general) return;
    const int x0 = blockIdx.x * kSegTX, tid = threadIdx.x;
    const size_t row = (size_t)blockIdx.y * W;
    auto lr = [](uint2 a) { return __byte_perm(a.x, a.y, 0x5410); };
    for (int i = tid; i < kSegTX + D - 1; i += 256) {
        int xt = x0 - D + 1 + i;
        if (xt < 0) xt += W;  // D <= W
        tar[i] = lr(ta[row + imin(xt, W - 1)]);
    }
    if (tid < kSegTX) ref[tid] = lr(ra[row + imin(x0 + tid, W - 1)]);
    __syncthreads();
    const int n = imin(kSegTX, W - x0) * D, half = kSegTX / 2 * D;
    const float *prow = pre + row * D;
    float *srow = seg + (row + x0) * D;
    for (int i = tid; i < n; i += 256) {
        const int up = i >= half ? kSegTX / 2 : 0, k = i - (up ? half : 0);
        const int px = (int)(((uint32_t)k * magic) >> 20), d = k - px * D, x = px + up;
        const uint32_t a = __vminu2(ref[x], tar[x + D - 1 - d]);
        const int xr = x0 + x + (int)(a >> 16), xl = imax(x0 + x - (int)(a & 0xffff) - 1, 0);  // :153-154
        srow[i] = __fsub_rn(prow[(size_t)xr * D + d], prow[(size_t)xl * D + d]);
    }
}

// acc += v where the mask has the bit, as one predicated add
__device__ __forceinline__ void add_if_bit(float &acc, uint32_t m, uint32_t bit, float v) {
    asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %1, %2;\n\tsetp.ne.u32 p, t, 0;\n\t"
        "@p add.rn.f32 %0, %0, %3;\n\t}"
        : "+f"(acc)
        : "r"(m), "r"(bit), "f"(v));
}

// Vertical sums: a warp streams 32 disparities (lane = disparity) of one column down
// a strip of rows, or for D <= 16 (8) the disparities of 2 (4) neighbouring columns
// (1 << lcw lanes a column).  Every lane keeps two rings of its own in shared memory
// (schedule and depth: rts_vert_ring.h), so the warps never wait on one another:
//   segments  [group of 4 rows][lane][4]: one 16-byte load gives four rows
//   words     [row][lane]: running sum of l + r down the column (low half, mod 2^16) |
//             t << 16 | b << 24, the entry's vertical arms
// Rows enter four at a time, the next four rows' loads in flight meanwhile.  A step
// makes four output rows together: a row read from the ring is added to each sum whose
// arm [y - t, y + b] holds it (one bit mask per output, four independent chains, rows
// top to bottom for every output).  The pixel count is a difference of running sums.
// Bound: instruction issue (about 100 instructions per 32 entries at short arms).
constexpr int kVolWarps = 4;
__global__ void __launch_bounds__(kVolWarps * 32, 4)
    k_cross_vol(const float *__restrict__ seg, const uint2 *__restrict__ aref, const uint2 *__restrict__ atar,
                float *__restrict__ out, const int *__restrict__ general, int H, int W, int D, int R, int lcw) {
    constexpr int S = kVertStep, DEP = vert_lane_depth(kModArm);
    extern __shared__ __align__(16) unsigned char vsm[];
    if (*general) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4 *segr = reinterpret_cast<float4 *>(vsm) + warp * (DEP / 4) * 32 + lane;  // group g at [32 g]
    uint32_t *wrd = reinterpret_cast<uint32_t *>(vsm + (size_t)kVolWarps * DEP * 128) + warp * DEP * 32 + lane;
    const int nch = (D + 31) >> 5, item = blockIdx.x * kVolWarps + warp;
    const int xw = (item / nch) << (5 - lcw), xl = xw + (lane >> lcw);
    if (xw >= W) return;
    const int x = imin(xl, W - 1), d = 32 * (item % nch) + (lane & ((1 << lcw) - 1));
    const bool dok = d < D && xl < W;  // other lanes follow an entry (x, 0) and write nothing
    const int y0 = blockIdx.y * R, y1 = imin(H, y0 + R);
    const int ra = imax(0, y0 - kModArm), rb = imin(H, y1 + kModArm);
    int xt = x - (dok ? d : 0);
    if (xt < 0) xt += W;  // D <= W
    const size_t rowD = (size_t)W * D;
    const float *segp = seg + (size_t)ra * rowD + (size_t)x * D + (dok ? d : 0);
    const uint2 *refp = aref + (size_t)ra * W + x, *tarp = atar + (size_t)ra * W + xt;
    const int nrows = rb - ra;
    float pseg[S];
    uint2 ptar[S], pref[S];
    auto load_rows = [&](int i) {
        const bool all = S * (i + 1) <= nrows;  // else the last rows, and rows with empty arms past them
#pragma unroll
        for (int k = 0; k < S; k++) {
            const bool in = all || S * i + k < nrows;
            pref[k] = in ? __ldg(refp) : make_uint2(0u, 0u);
            ptar[k] = in ? __ldg(tarp) : make_uint2(0u, 0u);
            pseg[k] = in ? __ldg(segp) : 0.f;
            refp += W;
            tarp += W;
            segp += rowD;
        }
    };
    int ts = 0;        // ring slot of the next rows to enter
    uint32_t cnt = 0;  // running sum of l + r in the low half
    auto ingest = [&](int i) {
        uint32_t w[S];
#pragma unroll
        for (int k = 0; k < S; k++) {
            const uint32_t lt = __vminu2(pref[k].x, ptar[k].x), rbm = __vminu2(pref[k].y, ptar[k].y);
            cnt += lt + rbm;
            w[k] = __byte_perm(cnt, __byte_perm(lt, rbm, 0x0062), 0x5410);  // low half | t << 16 | b << 24
        }
#pragma unroll
        for (int k = 0; k < S; k++) wrd[32 * (ts + k)] = w[k];
        segr[8 * ts] = make_float4(pseg[0], pseg[1], pseg[2], pseg[3]);  // group ts / 4
        ts += S;
        if (ts == DEP) ts = 0;
        load_rows(i + 1);
    };
    wrd[32 * (DEP - 1)] = 0u;  // the running sum before row ra
    load_rows(0);
    const int T0 = vert_lane_first(y0, ra, kModArm);
    int i = 0;
    for (; i < T0 - 1; i++) ingest(i);
    constexpr uint32_t end = (uint32_t)DEP * 128u;  // ring bytes of a lane's words
    uint32_t at0 = (uint32_t)(y0 - ra) * 128u;      // byte offset of the step's first output row
    const unsigned char *wb = reinterpret_cast<const unsigned char *>(wrd);
    auto word = [&](uint32_t o) { return *reinterpret_cast<const uint32_t *>(wb + o); };
    float *op = out + (size_t)y0 * rowD + (size_t)x * D + d;
    for (int y = y0; y < y1; y += S, i++) {
        ingest(i);
        float acc[S];
        uint32_t cn[S], m[S];
        int st[S], ln[S];  // first row of the arm, from the step's first output row; its rows
#pragma unroll
        for (int j = 0; j < S; j++) {
            uint32_t at = at0 + 128u * j;
            at = min(at, at - end);  // the ring's wrap, by an unsigned minimum
            const uint32_t w = word(at), t = __byte_perm(w, 0, 0x4442), b = w >> 24;
            st[j] = j - (int)t;
            ln[j] = (int)(t + b) + 1;
            const uint32_t up = at + 128u * b, dn = at - 128u * t - 128u;  // rows y + b and y - t - 1
            cn[j] = ((word(min(up, up - end)) - word(min(dn, dn + end))) & 0xffffu) + (uint32_t)ln[j];
            acc[j] = 0.f;
        }
        // rows lo .. hi - 1 hold every lane's arms
        int lo = imin(imin(st[0], st[1]), imin(st[2], st[3]));
        int hi = imax(imax(st[0] + ln[0], st[1] + ln[1]), imax(st[2] + ln[2], st[3] + ln[3]));
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        int g = (int)(at0 >> 7) + lo;  // ring slot of row lo
        g = g < 0 ? g + DEP : g;
        g = g >= DEP ? g - DEP : g;
        const int base = lo - (g & 3);  // the aligned group's first row
#pragma unroll
        for (int j = 0; j < S; j++) asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(m[j]) : "r"(st[j] - base), "r"(ln[j]));
        const int ng = (hi - base + 3) >> 2;
        const float4 *gp = segr + 8 * (g & ~3), *const gend = segr + 8 * DEP;
        auto walk = [&](int n) {
            for (int q = 0; q < n; q++) {
                const float4 v = *gp;
#pragma unroll
                for (int j = 0; j < S; j++) {
                    add_if_bit(acc[j], m[j], 1u, v.x);
                    add_if_bit(acc[j], m[j], 2u, v.y);
                    add_if_bit(acc[j], m[j], 4u, v.z);
                    add_if_bit(acc[j], m[j], 8u, v.w);
                    m[j] >>= 4;
                }
                gp += 32;
                if (gp == gend) gp = segr;
            }
        };
        walk(imin(ng, 8));
        if (ng > 8) {
            // rows 32 .. of long arms (at most 2 L + 7 < 64 rows in all)
#pragma unroll
            for (int j = 0; j < S; j++) {
                const int f = st[j] - base - 32, f0 = imax(f, 0);
                asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(m[j]) : "r"(f0), "r"(imax(f + ln[j] - f0, 0)));
            }
            walk(ng - 8);
        }
#pragma unroll
        for (int j = 0; j < S; j++, op += rowD)
            if (dok && y + j < y1) *op = __fdiv_rn(acc[j], (float)cn[j]);
        at0 += 128u * S;
        at0 = min(at0, at0 - end);
    }
}

// Any arms, straight from the running sums; an item is (row, 256 entries).  ctl: null (always;
// a block per item), or {flag that says whether the other kernels left the work, next item}.
// With the flag most calls leave at once, so the blocks are as many as are resident (an empty
// launch of 1280x720, D = 64 takes 123 us with an item a block, 4 us so), each taking the next
// kAggrGrab items as it comes to them: the blocks in flight have to stay on neighbouring
// rows, which the reads of a cross share in L2 (1280x720, D = 64, arms up to 3 and 25: an item a block
// 969 and 6952 us, resident blocks that stride over all items 1283 and 9855).
// Bound: the two reads a row and entry.
constexpr uint32_t kAggrGrab = 4;
__global__ void __launch_bounds__(256) k_cross_aggr(const float *__restrict__ pre, float *__restrict__ out,
                                                    const int *__restrict__ hr, const int *__restrict__ ht,
                                                    const int *__restrict__ vr, const int *__restrict__ vt,
                                                    uint32_t *__restrict__ ctl, int H, int W, int D) {
    __shared__ uint32_t grab;
    if (ctl && !ctl[0]) return;
    const uint32_t WD = (uint32_t)W * (uint32_t)D, nb = (WD + 255) >> 8, items = (uint32_t)H * nb;  // W D < 2^31
    auto one = [&](uint32_t item) {
        const uint32_t row = item / nb, i = (item - row * nb) * 256 + threadIdx.x;
        if (i >= WD) return;
        const int y = (int)row, x = (int)(i / (uint32_t)D), d = (int)(i - (uint32_t)x * D);
        const int xt = tar_col(x, d, W, 1);
        const long p = (long)y * W + x, q = (long)y * W + xt;
        const int t = imin(vr[2 * p], vt[2 * q]);
        const int b = imin(vr[2 * p + 1], vt[2 * q + 1]);
        float sum = 0.f;
        int cnt = 0;
        for (int yy = y - t; yy <= y + b; yy++) {
            if (yy < 0 || yy >= H) continue;
            const long pr = (long)yy * W + x, pt = (long)yy * W + xt;
            const int l = imin(hr[2 * pr], ht[2 * pt]);
            const int r = imin(hr[2 * pr + 1], ht[2 * pt + 1]);
            int xl = x - l - 1, xrr = x + r;
            if (xl < 0) xl = 0;  // :153-156 the clamped pixel is excluded from the sum, still counted
            else if (xrr >= W) xrr = W - 1;
            if (xl >= 0 && xrr < W && xl < W && xrr >= 0) {  // :157, always true for arms made by findCross
                const float *row = pre + (size_t)yy * W * D + d;
                sum = __fadd_rn(sum, __fsub_rn(row[(size_t)xrr * D], row[(size_t)xl * D]));
                cnt += r + l + 1;
            }
        }
        out[(size_t)p * D + d] = __fdiv_rn(sum, (float)cnt);
    };
    if (!ctl) {
        one(blockIdx.x);
        return;
    }
    for (;;) {
        __syncthreads();  // the last grab is read
        if (threadIdx.x == 0) grab = atomicAdd(ctl + 1, kAggrGrab);
        __syncthreads();
        const uint32_t first = grab;
        if (first >= items) return;
        for (uint32_t item = first; item < items && item < first + kAggrGrab; item++) one(item);
    }
}

size_t cross_aggr_bytes(int H, int W, int D, int arm) {
    const size_t np = (size_t)H * W;
    return np * D < kModSmall || D <= 2 || arm > kModArm ? 0 : np * (4 * (size_t)D + 16) + 256;
}

int launch_cross_aggr(cudaStream_t s, const float *pre, float *out, const int *hr, const int *ht, const int *vr,
                      const int *vt, int H, int W, int D, void *work) {
    const int sms = sm_count();
    if (!work) {
        k_cross_aggr<<<(unsigned)((long)H * (((long)W * D + 255) / 256)), 256, 0, s>>>(pre, out, hr, ht, vr, vt, nullptr,
                                                                                       H, W, D);
        return 1;
    }
    // {flag, next item, pad to 256 bytes | arm words of both images | segments}
    const size_t np = (size_t)H * W;
    int *general = (int *)work;
    uint2 *ra = (uint2 *)((unsigned char *)work + 256), *ta = ra + np;
    float *seg = (float *)(ta + np);
    cudaMemsetAsync(general, 0, 2 * sizeof(int), s);
    k_cross_pack<<<dim3((W + 127) / 128, H), 128, 0, s>>>(hr, ht, vr, vt, ra, ta, general, H, W);
    k_cross_seg<<<dim3((W + kSegTX - 1) / kSegTX, H), 256, 0, s>>>(pre, ra, ta, seg, general, W, D,
                                                                 ((1u << 20) + D - 1) / D);
    // strips: about two waves of warps where the columns alone are fewer (a strip repeats
    // up to 2 kModArm rows of its neighbours), none shorter than 24 rows
    const int lcw = D <= 8 ? 3 : D <= 16 ? 4 : 5;
    const long warps = (long)((W + (32 >> lcw) - 1) >> (5 - lcw)) * ((D + 31) / 32);
    const int strips = (int)std::max(1L, std::min((2L * 16 * sms + warps - 1) / warps, (long)H / 24));
    const int R = (H + strips - 1) / strips;
    const size_t smem = (size_t)kVolWarps * vert_lane_depth(kModArm) * 256;
    cudaFuncSetAttribute(k_cross_vol, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_cross_vol<<<dim3((unsigned)((warps + kVolWarps - 1) / kVolWarps), (H + R - 1) / R), kVolWarps * 32, smem, s>>>(
        seg, ra, ta, out, general, H, W, D, R, lcw);
    int res = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&res, k_cross_aggr, 256, 0) != cudaSuccess || res < 1) res = 1;
    k_cross_aggr<<<(unsigned)(sms * res), 256, 0, s>>>(pre, out, hr, ht, vr, vt, (uint32_t *)general, H, W, D);
    return 4;
}

}  // namespace rts
