// rts_pipe.h -- fused per-view pipeline kernels (k_pipe.cu) used by
// rts_pipeline.cpp when the configuration has a fused path.
#pragma once

#include "rts_internal.h"

namespace rts {

// AD / census (<= 64-bit window) single or combined costs, computed on the fly
bool fast_costs(const rts_params &p);
// every cost is >= 0: absolute differences and distances, and 1 - exp(-c / lambda) of such a
// c for a positive lambda; not NCC, nor AD cut at a negative truncation (cross-based
// aggregation truncates the first cost).  The kernels then order costs by their bits and
// divide by a product and its correction; others compare signed keys and divide.
bool costs_nonneg(const rts_params &p);
// adaptive-weight aggregation (radius <= 16) has a fused per-view path
bool fused_supported(const rts_params &p, int H, int W);

// 16-byte per-pixel records: census code, packed RGB (rgb null: the gray in all channels)
rts_status prep_records(rts_ctx *c, const rts_params &p, int H, int W, const uint8_t *gray, const uint8_t *rgb,
                        uint4 *rec);
// cost volume [H][W][D] (float, or __half when half != 0), pitch values a pixel, from
// records; mirror: of the mirrored images (a right view: reference and target are the right
// and the left image's records; their codes are then the mirrored images' up to one fixed
// order of the bits, which no distance depends on)
rts_status cost_volume_fast(rts_ctx *c, const rts_params &p, int H, int W, const uint4 *rr, const uint4 *rt,
                            void *vol, int half, int pitch, int mirror);
// the cross-based pipeline runs over view tables (rts_views.h) when this holds
bool cross_fused_supported(const rts_params &p);
// ... and for a disparity range that is not a multiple of 8 when this holds (in the plain
// form, whichever form is asked for: the composed path has no other)
bool cross_ragged_supported(const rts_params &p);
// adaptive-weight aggregation + arg-min over a float (half == 0) or __half volume of
// `pitch` values a pixel; mirror: of the mirrored Lab images
rts_status aw_fused(rts_ctx *c, const rts_params &p, int H, int W, const void *vol, int half, int pitch, const uint8_t *labr,
                    const uint8_t *labt, int mirror, uint16_t *raw, int *row_last, float *cost_out);

}  // namespace rts
