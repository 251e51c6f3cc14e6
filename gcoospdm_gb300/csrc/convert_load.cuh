// convert_load.cuh -- loads of A's rows that need not start on 16 bytes, for
// the conversions (not installed).
#pragma once

#include "internal.cuh"

namespace gcoo {

// The segment's 4 columns of lane `lane` (zeros past the row's `valid`
// columns), by a whole warp. seg: the row's first element of the segment.
// AL: every row starts on 16 bytes (k % 4 == 0, A aligned). Otherwise the row
// is shifted against the 16-byte granules by a warp-uniform 0..3 floats: each
// lane loads one granule and takes the rest of its four columns from the next
// lane's (lane 31 loads a 33rd); granules that reach outside A are read float
// by float. LAST: A's last reader (a streaming load).
template <bool AL, bool LAST>
__device__ __forceinline__ float4 seg_load(const float *seg, int lane, int64_t valid, const float *A, const float *A_end)
{
    const auto load = [](const float *p) {
        const float4 *q = reinterpret_cast<const float4 *>(p);
        return LAST ? __ldcs(q) : __ldg(q);
    };
    if constexpr (AL)
        return lane * 4 < valid ? load(seg + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    const int shift = static_cast<int>((reinterpret_cast<uintptr_t>(seg) >> 2) & 3u);
    const float *base = seg - shift;
    const auto granule = [&](int i) {
        const float *p = base + 4 * i;
        if (4 * i - shift >= valid)
            return make_float4(0.f, 0.f, 0.f, 0.f);
        if (p >= A && p + 4 <= A_end)
            return load(p);
        const auto one = [&](const float *q) { return q >= A && q < A_end ? __ldg(q) : 0.0f; };
        return make_float4(one(p), one(p + 1), one(p + 2), one(p + 3));
    };
    const float4 t = granule(lane);
    float x[8] = {t.x, t.y, t.z, t.w, 0.f, 0.f, 0.f, 0.f};
    if (shift) { // warp-uniform
        const float4 last = lane == 31 ? granule(32) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float y0 = __shfl_down_sync(0xffffffffu, t.x, 1), y1 = __shfl_down_sync(0xffffffffu, t.y, 1),
                    y2 = __shfl_down_sync(0xffffffffu, t.z, 1);
        x[4] = lane == 31 ? last.x : y0;
        x[5] = lane == 31 ? last.y : y1;
        x[6] = lane == 31 ? last.z : y2;
    }
    if (shift & 1) {
#pragma unroll
        for (int i = 0; i < 7; ++i)
            x[i] = x[i + 1];
    }
    if (shift & 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            x[i] = x[i + 2];
    }
    const int64_t left = valid - 4 * lane;
    return make_float4(left > 0 ? x[0] : 0.f, left > 1 ? x[1] : 0.f, left > 2 ? x[2] : 0.f, left > 3 ? x[3] : 0.f);
}

} // namespace gcoo
