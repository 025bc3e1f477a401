// rts_vert_ring.h -- row rings of the vertical cross-aggregation kernels: depths,
// and the rows ingested before the first step.  Plain constexpr arithmetic, shared
// by the kernels and by the CPU tests that replay it (tests/test_vert_ring.py,
// tests/test_vert_lane_ring.py).
//
// Block rings (k_vert_views, k_batch.cu).  A block of 8 warps walks one column
// from row y0; the ring holds rows from ra = max(0, y0 - L).  Rows enter 8 at a
// time ("ticks"): in tick i warp w writes row ra + 8 i + w into slot (8 i + w) mod
// depth.  Step s (one barrier each) first ingests tick T0 - 1 + s, then warp w reads
// rows y0 + 8 s + w - L .. y0 + 8 s + w + L.  With one barrier per step a fast
// warp may ingest tick T0 + s (the next step's) while a slow warp still reads
// step s: the newest row then written and the oldest row still read must not
// share a slot.
//
// Lane rings (k_vert_dual, k_batch.cu; k_cross_vol, k_cross_mod.cu).  A lane alone writes and reads its ring,
// so nothing but its own program order matters.  Rows enter kVertStep at a time;
// step s (output rows y0 + 4 s .. + 3) first lets tick vert_lane_first - 1 + s in,
// then reads rows y - L - 1 (the running count before the arm) .. y + L of its
// outputs.
#pragma once

#ifndef __CUDACC__
#ifndef __host__
#define __host__
#endif
#ifndef __device__
#define __device__
#endif
#endif

namespace rts {

// Ticks ingested before step 0 reads: every row up to y0 + 7 + L is in the ring.
__host__ __device__ constexpr int vert_first_ticks(int y0, int ra, int L) { return (y0 + 8 + L - ra + 7) >> 3; }

// Ring depth in rows for arm length L.  The newest row a fast warp writes
// during step s is ra + 8 (T0 + s) + 7 and the oldest row a slow warp reads
// is y0 + 8 s - L; with T0 = vert_first_ticks they are at most 2L + 22 rows
// apart (y0 - ra a multiple of 8, e.g. a strip at the image top).  The ring
// holds 2L + 23 rows or more, in whole ticks: a multiple of 8 (so also even,
// and two-row blocks of the walk never straddle the wrap).
__host__ __device__ constexpr int vert_depth(int L) { return 8 * ((2 * L + 23 + 7) / 8); }

constexpr int kVertStep = 4;  // rows of a tick, output rows of a step

// Ticks in before step 0 reads: every row up to y0 + 3 + L has entered.
__host__ __device__ constexpr int vert_lane_first(int y0, int ra, int L) {
    return (y0 + kVertStep + L - ra + kVertStep - 1) / kVertStep;
}

// Depth in rows.  Newest row in at step s: ra + 4 (T0 + s) - 1 <= y0 + 4 s + L + 6 with
// T0 = vert_lane_first; oldest row read: y0 + 4 s - L - 1; so at most 2 L + 8 rows,
// rounded to whole ticks (groups of four rows never straddle the wrap).
__host__ __device__ constexpr int vert_lane_depth(int L) {
    return kVertStep * ((2 * L + 2 * kVertStep + kVertStep - 1) / kVertStep);
}

// log2 of the power of two that covers D disparities in chunks of 32 (D <= 256)
__host__ __device__ constexpr int vert_log_chunks(int D) { return D <= 32 ? 0 : D <= 64 ? 1 : D <= 128 ? 2 : 3; }

}  // namespace rts
