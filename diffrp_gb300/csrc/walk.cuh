// walk.cuh -- sums over the pixels of a triangle, by columns.
//
// The backward passes add, for every pixel, a few quads of floats to rows that
// belong to its triangle's vertices.  A warp that walks 32 columns down, one per
// lane, keeps the sums of the triangle its column is in as registers: a pixel
// costs one addition per value, and a row of floats in shared memory only where
// the column leaves the triangle.  32 such rows are then added by columns of the
// row array, and go out with one vector atomic per run of rows of one triangle.
// (Reducing the runs of one pixel row by shuffles instead takes log2(run) steps
// of shuffle, compare and add per value, for every pixel row.)
#pragma once
#include "drp_common.cuh"

namespace drp {

// Shared rows of Q quads and the triangle's vertex indices (an int4 after
// them); the pitch is an odd number of 16-byte units (no bank conflicts).
template <int Q>
struct WalkRows {
    static constexpr int kIds = 4 * Q, kPitch = 4 * Q + (Q % 2 == 0 ? 4 : 8);
    float row[32][kPitch];
};

// Adds the first n rows (n warp-uniform, at most 32): add(row, quad, sum) is
// called by the lane that holds a run's sum of one quad, with a row of the run.
// All 32 lanes call it, after they have written their rows.
template <int Q, class Add>
__device__ __forceinline__ void walk_drain(const WalkRows<Q>& sh, int n, const Add& add) {
    constexpr int PARTS = 32 / Q, LEN = (32 + PARTS - 1) / PARTS;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    int4 id = make_int4(-1, -1, -1, 0);
    if (lane < n) id = *reinterpret_cast<const int4*>(&sh.row[lane][WalkRows<Q>::kIds]);
    const int nx = __shfl_down_sync(0xffffffffu, id.x, 1), ny = __shfl_down_sync(0xffffffffu, id.y, 1),
              nz = __shfl_down_sync(0xffffffffu, id.z, 1);
    const unsigned ends = __ballot_sync(0xffffffffu, lane == 31 || nx != id.x || ny != id.y || nz != id.z);
    const int part = lane / Q, quad = lane - part * Q, first = part * LEN, len = min(n - first, LEN);
    if (part < PARTS && len > 0) {
        const unsigned my_ends = (ends >> first) | (1u << (len - 1));
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < LEN; ++k) {
            if (k >= len) break;
            const float* row = sh.row[first + k];
            const float4 x = *reinterpret_cast<const float4*>(row + 4 * quad);
            acc.x += x.x;
            acc.y += x.y;
            acc.z += x.z;
            acc.w += x.w;
            if ((my_ends >> k) & 1u) {
                add(row, quad, acc);
                acc = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    __syncwarp();
}

// One step of a walk: the lanes whose column enters another triangle put the
// sums of the one they leave into the next rows (leave(row)), after a drain
// when there is no room.  n: rows in use.  All 32 lanes call it.
template <int Q, class Leave, class Add>
__device__ __forceinline__ void walk_leave(WalkRows<Q>& sh, int& n, bool leaves, const Leave& leave, const Add& add) {
    const unsigned m = __ballot_sync(0xffffffffu, leaves);
    if (!m) return;
    if (n + __popc(m) > 32) {
        walk_drain<Q>(sh, n, add);
        n = 0;
    }
    if (leaves) leave(sh.row[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))]);
    n += __popc(m);
}

// Columns, rows and view of a warp's strip of a (B, H, W) image: 32 columns x
// `rows` rows.
constexpr int kWalkWarps = 4;
struct WalkStrip {
    int b, x0, y0, y1;
};
__device__ __forceinline__ bool walk_strip(int B, int H, int W, int rows, WalkStrip& s) {
    const int ux = (W + 31) / 32, uy = (H + rows - 1) / rows;
    const long long unit = (long long)blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
    const long long row = unit / ux;
    s.b = (int)(row / uy);
    if (s.b >= B) return false;
    s.x0 = 32 * (int)(unit - row * ux);
    s.y0 = rows * (int)(row - (long long)s.b * uy);
    s.y1 = min(s.y0 + rows, H);
    return true;
}
inline unsigned walk_blocks(int B, int H, int W, int rows) {
    const long long units = (long long)B * ((W + 31) / 32) * ((H + rows - 1) / rows);
    return (unsigned)((units + kWalkWarps - 1) / kWalkWarps);
}

}  // namespace drp
