// batch.cu -- the batching form: many meshes x views x resolutions in one
// set of launches, with raster + interpolation fused and the whole backward
// (antialias, interpolation, rasterisation) fused into one pixel pass.
//
// An item is one (mesh, view, resolution) render: its clip vertices, its
// mesh's triangles and attributes, and its own output image.  All items'
// data live in packed buffers addressed through a device item table
// (drp_batch_item); host-built block maps send every 256-wide block of
// primitives or pixels to one item, so no thread searches for its item.
//
// Forward launches (independent of the number of items):
//   setup/count -> scan -> setup/fill  (tile lists for every item's tiles)
//   fine raster: persistent CTAs pull (item, tile) work from an atomic queue,
//                resolve visibility, write rast and the interpolated colour
//   antialias:   per-triangle records, then the per-pixel silhouette blend
// Backward: per-triangle records, then one fused pixel pass computing the
// antialias colour gradient, the attribute gradient (interpolation backward)
// and the vertex gradient (rasterisation backward), scattered with
// warp-segmented float4 atomics.
#include <atomic>

#include "../../include/diffrp_gb300.h"
#include "aa_core.cuh"
#include "drp_internal.h"
#include "raster_core.cuh"

namespace drp {

struct BatchArgs {
    const drp_batch_item* items;
    int num_items;
    const int2* prim_blocks;  // (item, local block) per 256 triangle slots
    long long n_prim_blocks;
    const int2* pix_blocks;   // (item, local block) per 256 pixels
    long long n_pix_blocks;
    long long total_prims, total_tiles;
    long long total_pixels;  // drp_batch_render
    const float* pos;
    const int* tri;
    const float* attr;
    const int* nbr;
    int tile_log2, tpt;
    unsigned long long list_capacity;
    uint32_t bin_depth;  // 0: exact lists (count, scan, fill); > 0: fixed-depth bins (one pass)
    float* rast;
    float* color;
    float* out;
    // antialias state (forward writes, backward reads): per pixel whether a
    // blending pair touches it, and the list of those pixels
    unsigned char* aa_flags;
    int* aa_list;
    unsigned* aa_count;
    bool fit;               // the fine raster writes the pixel words, for batch_fit_kernel or batch_blend_kernel
    uint32_t* aa_words;     // per pixel: triangle + 1 (0: none), kPixSil where its record has a silhouette edge
    bool emit_color;        // fit: the fine raster writes the colour of every pixel
    bool emit_out;          // the fine raster also writes the colour into out
    bool aa_records;        // the setup pass writes the antialias triangle records
    // fused mean-absolute-error loss (null target: none)
    const float* target;
    float l1_scale;
    float* l1_grad;
    float* block_loss;      // one partial per pixel block
    float* loss;
    bool l1_grads;          // the loss pass also forms the loss's gradient (drp_batch_forward_l1_grad)
    float* zero_first;      // floats zeroed by the forward's first kernel (null: none)
    long long zero_floats;
    const float* grad_scale;  // backward: device scalar multiplying grad_out, or null
    const float* grad_out;
    float* grad_pos;
    float* grad_attr;
    // workspace
    uint32_t* stats;
    uint32_t* queue;
    uint32_t* loss_count;  // CTAs of the list kernel that have added their slice of the loss
    int4* prims;
    uint32_t *tile_count, *tile_offset, *tile_cursor, *tile_list;
    unsigned long long* chunk_sums;  // tile-scan chunk sums
    float4* aa_rec;
    const uint32_t* tile_order = nullptr;  // fine-raster work order (null: tile index order)
};

// MODE kSetupCount: triangle setup, antialias record, per-tile counts;
// kSetupFill: append to the exact lists (after the scan); kSetupBins: setup,
// record and append to fixed-depth bins in one pass.
constexpr int kSetupCount = 0, kSetupFill = 1, kSetupBins = 2;
// CTAs per 256-triangle block of the map: the work is a chain of dependent
// loads per triangle, so smaller CTAs spread one mesh's few hundred map blocks
// over every SM.  The fill's chain is short and large meshes wait for its CTAs to
// start: two blocks of 128 triangles instead of four of 64 take 101 instead of
// 135 us for four views of 2.09M triangles and 167 instead of 248 for 16 of 980k
// (the count pass with two: 395 against 383, 679 against 654).
__host__ __device__ constexpr int setup_split(int mode) { return mode == kSetupFill ? 2 : 4; }
constexpr int kSetupSplitMost = 4;

template <int TILE_LOG2, int MODE>
__global__ void __launch_bounds__(2 * 256 / setup_split(MODE)) batch_setup_bin_kernel(BatchArgs a) {
    constexpr int kSetupSplit = setup_split(MODE), kSetupTris = 256 / kSetupSplit;
    pdl_wait();
    pdl_launch_dependents();
    constexpr bool FILL = MODE == kSetupFill;
    const int2 blk = a.prim_blocks[blockIdx.x / kSetupSplit];
    const drp_batch_item& it = a.items[blk.x];
    const long long j0 = (long long)blk.y * 256 + (blockIdx.x % kSetupSplit) * kSetupTris;
    // Count / bin launches with antialias records use 2 * kSetupTris threads:
    // the upper half writes the records of the CTA's triangles while the
    // lower half sets them up and bins them (two shorter chains of dependent
    // loads instead of one).  Whole warps take one side.
    if (threadIdx.x >= kSetupTris) {
        const long long jr = j0 + (threadIdx.x - kSetupTris);
        if (!FILL && a.aa_records && jr < it.tri_count)
            aa_tri_record(reinterpret_cast<const float4*>(a.pos) + it.pos_offset,
                          a.tri + 3 * (long long)it.tri_first, a.nbr ? a.nbr + 3 * (long long)it.tri_first : nullptr,
                          jr, it.tri_count, it.num_vertices, it.width, it.height,
                          a.aa_rec + (it.prim_offset + jr) * 2);
        return;
    }
    // every lane stays to the binning (a warp-collective call)
    const long long j = j0 + threadIdx.x;
    const bool in = j < it.tri_count;
    const long long pidx = it.prim_offset + (in ? j : 0);
    int4* rec = a.prims + pidx * 3;
    PrimBox bx;
    bx.px0 = 1;
    bx.px1 = bx.py0 = bx.py1 = 0;
    bool live = false;
    if (FILL) {
        if (in) {
            bx = unpack_box(rec[1], rec[2]);
            live = bx.px0 <= bx.px1;
        }
    } else if (in) {
        const long long t = (long long)it.tri_first + j;
        const int i0 = a.tri[3 * t], i1 = a.tri[3 * t + 1], i2 = a.tri[3 * t + 2];
        if (i0 < 0 || i1 < 0 || i2 < 0 || i0 >= it.num_vertices || i1 >= it.num_vertices || i2 >= it.num_vertices) {
            atomicOr(a.stats + 2, DRP_DEVERR_BAD_INDEX);
        } else {
            const float4* P = reinterpret_cast<const float4*>(a.pos) + it.pos_offset;
            live = build_prim(P[i0], P[i1], P[i2], j, it.width, it.height, rec, bx);
        }
        if (!live) {
            rec[0] = make_int4(0, 0, 0, 0);
            rec[1] = make_int4(0, 0, 0, 1);
            rec[2] = make_int4(0, 0, 0, 0);
        }
    }
    if (FILL) {
        bin_box<TILE_LOG2>(bx, live, it.tiles_x, a.tile_cursor + it.tile_offset, a.tile_list, a.list_capacity,
                           (uint32_t)pidx);
    } else {
        if (MODE == kSetupBins)
            bin_box<TILE_LOG2>(bx, live, it.tiles_x, a.tile_count + it.tile_offset,
                               a.tile_list + (unsigned long long)it.tile_offset * a.bin_depth, 0, (uint32_t)pidx,
                               a.bin_depth);
        else
            bin_box<TILE_LOG2>(bx, live, it.tiles_x, a.tile_count + it.tile_offset, nullptr, 0, 0);
    }
}

// rast + interpolated attributes of one pixel (interpolator.py:45 order).
// The colour also goes to out (when not null): the antialias pass then only
// rewrites the pixels it blends.
template <bool FIT>
struct BatchEmit {
    const float4* P;
    const int* tri;  // the item's mesh triangles (local vertex indices)
    const float* A;  // the item's mesh attributes
    int W, H, C;
    bool vec;  // 128-bit attribute / colour / output access: C % 4 == 0 and all bases 16-byte aligned
    float4* rast;
    float* color;       // FIT: null where only the listed pixels' colours are wanted
    float* out;
    uint32_t* words;    // FIT: the item's pixel words
    const float4* rec;  // FIT: the item's antialias records
    __device__ __forceinline__ void operator()(int px, int py, unsigned long long k, float X, float Y) const {
        const long long o = (long long)py * W + px;
        float* col = color + o * C;
        float* oc = out ? out + o * C : nullptr;
        if (k == ~0ull) {
            rast[o] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (FIT) {
                words[o] = 0u;
                if (!color) return;
            }
            if (vec) {
                for (int c = 0; c < C; c += 4) {
                    *reinterpret_cast<float4*>(col + c) = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (oc) *reinterpret_cast<float4*>(oc + c) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            } else {
                for (int c = 0; c < C; ++c) {
                    col[c] = 0.f;
                    if (oc) oc[c] = 0.f;
                }
            }
            return;
        }
        const int t = (int)(uint32_t)(k & 0xffffffffu);
        const int i0 = tri[3 * (long long)t], i1 = tri[3 * (long long)t + 1], i2 = tri[3 * (long long)t + 2];
        Shade S;
        shade_eval_xy(P[i0], P[i1], P[i2], X, Y, W, H, S);
        rast[o] = make_float4(S.u, S.v, S.zw, enc_triid(t + 1));
        if (FIT) {
            words[o] = (uint32_t)(t + 1) | (__float_as_uint(rec[2 * (long long)t + 1].w) ? kPixSil : 0u);
            if (!color) return;
        }
        const float* a0 = A + (long long)i0 * C;
        const float* a1 = A + (long long)i1 * C;
        const float* a2 = A + (long long)i2 * C;
        if (vec) {
            for (int c = 0; c < C; c += 4) {
                const float4 x0 = __ldg(reinterpret_cast<const float4*>(a0 + c));
                const float4 x1 = __ldg(reinterpret_cast<const float4*>(a1 + c));
                const float4 x2 = __ldg(reinterpret_cast<const float4*>(a2 + c));
                float4 o;
                o.x = fmaf(x0.x - x2.x, S.u, fmaf(x1.x - x2.x, S.v, x2.x));
                o.y = fmaf(x0.y - x2.y, S.u, fmaf(x1.y - x2.y, S.v, x2.y));
                o.z = fmaf(x0.z - x2.z, S.u, fmaf(x1.z - x2.z, S.v, x2.z));
                o.w = fmaf(x0.w - x2.w, S.u, fmaf(x1.w - x2.w, S.v, x2.w));
                *reinterpret_cast<float4*>(col + c) = o;
                if (oc) *reinterpret_cast<float4*>(oc + c) = o;
            }
        } else {
            for (int c = 0; c < C; ++c) {
                const float v = fmaf(a0[c] - a2[c], S.u, fmaf(a1[c] - a2[c], S.v, a2[c]));
                col[c] = v;
                if (oc) oc[c] = v;
            }
        }
    }
};

__device__ __forceinline__ int find_item_by_tile(const drp_batch_item* items, int n, long long tile) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (items[mid].tile_offset <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <int TILE_LOG2, int TPT, bool FIT, int NT>
__global__ void __launch_bounds__(NT, fine_ctas<TILE_LOG2, NT>())
batch_fine_kernel(BatchArgs a) {
    // The tile's parameters live in shared memory, filled by thread 0 with
    // the job: held in registers through the fine raster they pushed its
    // working set past the 64 registers of 4 CTAs per SM (spills).
    __shared__ long long job;
    __shared__ FineTile ft;
    __shared__ BatchEmit<FIT> e;
    pdl_wait();
    pdl_launch_dependents();
    for (;;) {
        __syncthreads();  // every thread is done with the previous tile's job, ft and e
        if (threadIdx.x == 0) {
            const long long j = (long long)atomicAdd(a.queue, 1u);
            const long long t = j < a.total_tiles && a.tile_order ? (long long)a.tile_order[j] : j;
            job = t;
            if (t < a.total_tiles) {
                const int ii = find_item_by_tile(a.items, a.num_items, t);
                const drp_batch_item& it = a.items[ii];
                const int tile = (int)(t - it.tile_offset);
                ft.recs = a.prims;
                ft.cnt = a.tile_count[t];
                if (a.bin_depth) {
                    ft.list = a.tile_list + (unsigned long long)t * a.bin_depth;
                    ft.overflow = ft.cnt > a.bin_depth;
                    if (ft.overflow) atomicMax(a.stats + 3, ft.cnt);  // sizes the next depth
                } else {
                    const uint32_t off = a.tile_offset[t];
                    ft.list = a.tile_list + off;
                    ft.overflow = (unsigned long long)off + ft.cnt > a.list_capacity;
                }
                ft.scan_base = it.prim_offset;
                ft.scan_count = it.tri_count;
                ft.tx0 = (tile % it.tiles_x) << TILE_LOG2;
                ft.ty0 = (tile / it.tiles_x) << TILE_LOG2;
                ft.W = it.width;
                ft.H = it.height;
                ft.P = reinterpret_cast<const float4*>(a.pos) + it.pos_offset;
                ft.tri = a.tri + 3 * (long long)it.tri_first;
                ft.prev = nullptr;
                ft.stats = a.stats;
                e.P = ft.P;
                e.tri = ft.tri;
                e.A = a.attr + it.attr_offset;
                e.W = it.width;
                e.H = it.height;
                e.C = it.channels;
                e.rast = reinterpret_cast<float4*>(a.rast) + it.pixel_offset;
                e.color = !FIT || a.emit_color ? a.color + it.image_offset : nullptr;
                e.out = a.emit_out ? a.out + it.image_offset : nullptr;
                if (FIT) {
                    e.words = a.aa_words + it.pixel_offset;
                    e.rec = a.aa_rec + it.prim_offset * 2;
                }
                e.vec = (it.channels & 3) == 0 &&
                        ((reinterpret_cast<uintptr_t>(e.A) | reinterpret_cast<uintptr_t>(e.color) |
                          reinterpret_cast<uintptr_t>(e.out)) & 15) == 0;
            }
        }
        __syncthreads();
        if (job >= a.total_tiles) break;
        fine_tile<TILE_LOG2, TPT, false, NT>(ft, e);
    }
}

__global__ void __launch_bounds__(256) batch_aa_setup_kernel(BatchArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    const int2 blk = a.prim_blocks[blockIdx.x];
    const drp_batch_item& it = a.items[blk.x];
    const long long j = (long long)blk.y * 256 + threadIdx.x;
    if (j >= it.tri_count) return;
    const float4* P = reinterpret_cast<const float4*>(a.pos) + it.pos_offset;
    aa_tri_record(P, a.tri + 3 * (long long)it.tri_first, a.nbr ? a.nbr + 3 * (long long)it.tri_first : nullptr, j,
                  it.tri_count, it.num_vertices, it.width, it.height, a.aa_rec + (it.prim_offset + j) * 2);
}

// Record a pixel some blending pair touches: its flag, and (warp-aggregated)
// its global index in the list the antialias backward walks.  All 32 lanes
// of the warp call it.
// FLAGS = false: the list only (the forward that forms the loss's gradient
// has no backward pass to read the per-pixel flags).
template <bool FLAGS = true>
__device__ __forceinline__ void aa_note_pixel(const BatchArgs& a, long long gpix, bool in, unsigned bits) {
    if (!a.aa_flags) return;
    if (FLAGS && in) a.aa_flags[gpix] = bits ? 1 : 0;
    const bool need = in && bits != 0u;
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(a.aa_count, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (need) a.aa_list[base + __popc(m & ((1u << lane) - 1u))] = (int)gpix;
}

__global__ void __launch_bounds__(256) batch_aa_fwd_kernel(BatchArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    const int2 blk = a.pix_blocks[blockIdx.x];
    const drp_batch_item& it = a.items[blk.x];
    const int pix = blk.y * 256 + threadIdx.x;
    const bool in = pix < it.width * it.height;
    unsigned bits = 0;
    if (in) {
        const float4* R = reinterpret_cast<const float4*>(a.rast) + it.pixel_offset;
        // out already holds the colour (written by the fine raster): only blended pixels change
        aa_fwd_pixel<false>(R, a.color + it.image_offset, a.aa_rec + it.prim_offset * 2, it.tri_count, it.width,
                            it.height, it.channels, pix, a.out + it.image_offset + (long long)pix * it.channels,
                            &bits);
    }
    aa_note_pixel(a, it.pixel_offset + pix, in, bits);
}

// Antialias forward with the mean-absolute-error loss fused: every pixel's
// output (written when out is set), sign gradient and |error| sum; one
// partial per 256-pixel block, added in index order by the final reduction
// (reproducible loss).
__global__ void __launch_bounds__(256, 5) batch_aa_l1_kernel(BatchArgs a) {
    __shared__ float warp_sum[8];
    pdl_wait();
    pdl_launch_dependents();
    const int2 blk = a.pix_blocks[blockIdx.x];
    const drp_batch_item& it = a.items[blk.x];
    const int pix = blk.y * 256 + threadIdx.x;
    float s = 0.0f;
    const bool in = pix < it.width * it.height;
    unsigned bits = 0;
    {
        const float4* R = reinterpret_cast<const float4*>(a.rast) + it.pixel_offset;
        int src[4];
        float wt[4];
        const bool any = aa_fwd_terms_row(R, a.aa_rec + it.prim_offset * 2, it.tri_count, it.width, it.height, pix,
                                          in, src, wt, &bits);  // all lanes: pairs shared along the row
        if (in) {
            const long long row = it.image_offset + (long long)pix * it.channels;
            s = aa_l1_channels(a.color + it.image_offset, it.channels, pix, src, wt, any, a.target + row,
                               a.l1_scale, a.out ? a.out + row : nullptr, a.l1_grad + row);
        }
    }
    aa_note_pixel(a, it.pixel_offset + pix, in, bits);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += warp_sum[w];
        a.block_loss[blockIdx.x] = t;
    }
}

__device__ __forceinline__ int find_item_by_pixel(const drp_batch_item* items, int n, long long gpix) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (items[mid].pixel_offset <= gpix) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Whole backward of the listed pixels (those a blending pair touches, about
// the silhouettes): edge-vertex gradients (scattered once per pair by its
// first pixel), the pixel's antialiased colour gradient, and with it the
// pixel's interpolation backward (attribute atomics) and rasterisation
// backward (vertex atomics).  batch_bwd_kernel skips these pixels, so the two
// kernels are independent and run side by side.  The list is short and each
// pixel's chain of dependent loads is long, so a group of LANES lanes takes
// one pixel: lane q evaluates pair slots q, q + LANES, ... (and scatters a
// slot's edge gradient when it owns the pair), the group exchanges the slot
// terms by shuffles, the lanes share the channels (c = q, q + LANES, ...) and
// sum d/du, d/dv by shuffles.  Grid-stride over the device-side count, so
// the launch needs no host sync; the grid is one resident wave
// (list_kernel_grid).  L1G (the forward that forms the loss's gradient): the
// kernel follows the antialias / loss pass on the launch chain and forms the
// loss before its pixels, without a separate final-sum launch: its last block
// from batch_aa_l1_grad_kernel's partials, or every block a slice of
// batch_fit_kernel's region sums (fit_loss).
// The incoming image gradient of one item: the gradient buffer times the
// upstream scale, or (L1G, the forward that forms the loss's gradient) the
// L1 sign gradient from the output and the target.
template <bool L1G>
struct ItemGrad;
template <>
struct ItemGrad<false> {
    static __device__ __forceinline__ GradBuffer of(const BatchArgs& a, const drp_batch_item& it, float gsc) {
        return GradBuffer{a.grad_out + it.image_offset, gsc};
    }
};
template <>
struct ItemGrad<true> {
    static __device__ __forceinline__ GradL1 of(const BatchArgs& a, const drp_batch_item& it, float) {
        return GradL1{a.out + it.image_offset, a.target + it.image_offset, a.l1_scale};
    }
};

// Launches of at least this many pixels may form the loss and its gradient with
// batch_fit_kernel (fit_words_bytes); the others take batch_aa_l1_grad_kernel, whose
// shorter chain per pixel is what counts while the regions fill only part of the
// chip: one view of 400 x 400 takes 58.5 with the first against 55.3 us per step with
// the second at 3 channels and 68.2 against 63.8 at 8.
constexpr long long kFitPixels = 1ll << 20;

// batch_fit_kernel takes regions of 32 x 16 pixels, a fixed number per raster
// tile in grid order: the halves of a 32-pixel tile, a pair of 16-pixel tiles
// or a 4 x 2 block of 8-pixel ones (their first tile takes it, the others
// nothing).  Region i leaves its |error| sum in a tile word the raster has
// spent: the tile's list offset, or for the second half its cursor.
__host__ __device__ inline int fit_regions_per_tile(int tile_log2) { return tile_log2 == 5 ? 2 : 1; }

__device__ __forceinline__ bool fit_region_owner(int tile_log2, int tx, int ty) {
    return tile_log2 == 5 || (tile_log2 == 4 ? (tx & 1) == 0 : (tx & 3) == 0 && (ty & 1) == 0);
}

__device__ __forceinline__ float* fit_loss_slot(const BatchArgs& a, long long i) {
    if (a.tile_log2 != 5) return reinterpret_cast<float*>(a.tile_offset + i);
    return reinterpret_cast<float*>(((i & 1) ? a.tile_cursor : a.tile_offset) + (i >> 1));
}

// The loss from the regions' sums: every CTA adds a contiguous slice of them
// and leaves its sum in the slice's first slot and the sum's error in the second
// (a slice of one has none); the CTA that arrives last (a counter the forward's
// first kernel zeroed; nobody waits) adds the slices.  Fixed slices, fixed order
// within each: reproducible.  One CTA adding every partial took 27 us of the
// 64-view step.
__device__ __forceinline__ void fit_loss(const BatchArgs& a) {
    __shared__ bool last;
    const long long n = a.total_tiles * fit_regions_per_tile(a.tile_log2);
    const long long per = (n + gridDim.x - 1) / gridDim.x;
    const long long b0 = blockIdx.x * per, b1 = b0 + per < n ? b0 + per : n;
    float s = 0.f, c = 0.f;
    for (long long i = b0 + threadIdx.x; i < b1; i += blockDim.x) two_sum(s, c, *fit_loss_slot(a, i));
    const float2 slice = block_sum_pairs<kFinalThreads>(s, c);
    if (threadIdx.x == 0) {
        if (b0 < b1) *fit_loss_slot(a, b0) = slice.x;
        if (b0 + 1 < b1) *fit_loss_slot(a, b0 + 1) = slice.y;
        __threadfence();
        last = atomicAdd(a.loss_count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = c = 0.f;
    for (long long b = threadIdx.x * per; b < n; b += blockDim.x * per) {
        two_sum(s, c, __ldcg(fit_loss_slot(a, b)));
        if (per > 1 && b + 1 < n) c += __ldcg(fit_loss_slot(a, b + 1));
    }
    const float2 sum = block_sum_pairs<kFinalThreads>(s, c);
    if (threadIdx.x == 0) *a.loss = (sum.x + sum.y) * a.l1_scale;
}

// Lanes per listed pixel in batch_aa_bwd_kernel.  Two lanes cover twice the
// pixels of four per resident wave (the single-mesh step lists ~45K pixels:
// one wave with two, two with four), but each lane's chain of slot
// evaluations doubles and the kernel needs 74 registers; four measured
// slightly faster on the single-mesh step (157.1 vs 159.2 us per step).
#ifndef DRP_LIST_LANES
#define DRP_LIST_LANES 4
#endif
constexpr int kListLanes = DRP_LIST_LANES;

// Who launches it: the ordinary backward, or the forward that forms the loss's
// gradient, after batch_aa_l1_grad_kernel or batch_fit_kernel.  (The two sums
// of the loss are separate instantiations: with both in one the list of small
// launches took 16.5 instead of 15.8 us, one view of 256 x 256 x 3.)
constexpr int kListBackward = 0, kListL1 = 1, kListFit = 2;

template <int KIND, int LANES>
__global__ void __launch_bounds__(256, KIND == kListL1 ? 0 : 3) batch_aa_bwd_kernel(BatchArgs a) {
    constexpr bool L1G = KIND != kListBackward;
    static_assert(LANES == 2 || LANES == 4, "two or four lanes per listed pixel");
    constexpr int SLOTS = 4 / LANES;  // pair slots each lane evaluates
    pdl_wait();
    pdl_launch_dependents();
    static_assert(kFinalThreads == 256, "the list kernel's blocks form the loss");
    if (KIND == kListFit)
        fit_loss(a);
    else if (KIND == kListL1 && blockIdx.x == gridDim.x - 1)
        l1_final_block<kFinalThreads>(a.block_loss, a.n_pix_blocks, a.l1_scale, a.loss);
    const unsigned n = *a.aa_count;
    const float gsc = (!L1G && a.grad_scale) ? *a.grad_scale : 1.0f;
    const int lane = threadIdx.x & 31, q = lane & (LANES - 1), qbase = lane & ~(LANES - 1);
    const long long groups = ((long long)gridDim.x * blockDim.x) / LANES;
    for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;; i += groups) {
        const bool active = i < n;
        if (!__any_sync(0xffffffffu, active)) break;  // warp-uniform exit (lane groups step together)
        int role[SLOTS], tgt[SLOTS], pix = 0, C = 0;
        float wt[SLOTS];
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            role[j] = 0;
            tgt[j] = 0;
            wt[j] = 0.f;
        }
        const drp_batch_item* itp = nullptr;
        if (active) {
            const long long gpix = a.aa_list[i];
            itp = &a.items[find_item_by_pixel(a.items, a.num_items, gpix)];
            const drp_batch_item& it = *itp;
            pix = (int)(gpix - it.pixel_offset);
            C = it.channels;
            const int W = it.width, H = it.height;
            const int py = pix / W, px = pix - py * W;
            const float4* R = reinterpret_cast<const float4*>(a.rast) + it.pixel_offset;
            const float4 rs = R[pix];
#pragma unroll
            for (int j = 0; j < SLOTS; ++j) {
                int A, B, ax, ay;
                bool vert;
                if (!pair_slot(q + j * LANES, pix, px, py, W, H, A, B, ax, ay, vert)) continue;
                const float4 ro = R[A == pix ? B : A];
                if (ro.w == rs.w) continue;
                AAPair p;
                aa_pair(a.aa_rec + it.prim_offset * 2, it.tri_count, A, B, ax, ay, vert, A == pix ? rs : ro,
                        A == pix ? ro : rs, p);
                if (!p.valid) continue;
                role[j] = p.target == pix ? 1 : 2;
                tgt[j] = p.target;
                wt[j] = p.w;
                if (A == pix && !p.clamped)
                    aa_edge_grad_g(p, a.color + it.image_offset, ItemGrad<L1G>::of(a, it, gsc), C,
                                   reinterpret_cast<const float4*>(a.pos) + it.pos_offset,
                                   a.tri + 3 * (long long)it.tri_first,
                                   reinterpret_cast<float4*>(a.grad_pos) + it.pos_offset, 1.0f, W, H);
            }
        }
        // slot k was evaluated by lane (k % LANES) of the group, as its
        // (k / LANES)-th slot
        AATerms at;
        at.any = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int src = qbase | (k % LANES);
            at.role[k] = __shfl_sync(0xffffffffu, role[k / LANES], src);
            at.tgt[k] = __shfl_sync(0xffffffffu, tgt[k / LANES], src);
            at.wt[k] = __shfl_sync(0xffffffffu, wt[k / LANES], src);
            at.any = at.any || at.role[k] != 0;
        }
        int t = -1, i0 = 0, i1 = 0, i2 = 0;
        float gu = 0.f, gv = 0.f;
        if (active) {
            const drp_batch_item& it = *itp;
            const int* tri = a.tri + 3 * (long long)it.tri_first;
            const float4 r = reinterpret_cast<const float4*>(a.rast)[it.pixel_offset + pix];
            t = checked_tri(r.w, tri, it.tri_count, it.num_vertices, i0, i1, i2);
            if (t >= 0) {
                const auto grad = ItemGrad<L1G>::of(a, it, gsc);
                const float* A = a.attr + it.attr_offset;
                float* GA = a.grad_attr + it.attr_offset;
                const float u = r.x, v = r.y, w = 1.0f - u - v;
                // Channels four to a lane where that leaves two lanes work (one for
                // four channels: 154 -> 158 us on 16 dense 512 x 512 views): a
                // quarter of the atomics.  Eight channels 109 -> 102 us (64 views),
                // 16 channels 41 -> 37 us (one 1024 x 1024 view).  Small launches
                // (kListL1) wait for the longest chain, not the atomics: the code's
                // registers cost the smallest step 0.2 us.
                if (KIND != kListL1 && (C & 3) == 0 && C >= 8 && grad.aligned() &&
                    ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(GA)) & 15) == 0) {
                    for (int c = 4 * q; c < C; c += 4 * LANES) {
                        const float4 g4 = grad.load4((long long)pix * C + c);
                        float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            if (at.role[k] == 0) continue;
                            const bool own = at.role[k] == 1;
                            const float4 n4 = own ? g4 : grad.load4((long long)at.tgt[k] * C + c);
                            const float wk = own ? -at.wt[k] : at.wt[k];
                            g[0] = fmaf(wk, n4.x, g[0]);
                            g[1] = fmaf(wk, n4.y, g[1]);
                            g[2] = fmaf(wk, n4.z, g[2]);
                            g[3] = fmaf(wk, n4.w, g[3]);
                        }
                        const float4 x0 = *reinterpret_cast<const float4*>(A + (long long)i0 * C + c);
                        const float4 x1 = *reinterpret_cast<const float4*>(A + (long long)i1 * C + c);
                        const float4 x2 = *reinterpret_cast<const float4*>(A + (long long)i2 * C + c);
                        atomic_add4(reinterpret_cast<float4*>(GA + (long long)i0 * C + c),
                                    make_float4(g[0] * u, g[1] * u, g[2] * u, g[3] * u));
                        atomic_add4(reinterpret_cast<float4*>(GA + (long long)i1 * C + c),
                                    make_float4(g[0] * v, g[1] * v, g[2] * v, g[3] * v));
                        atomic_add4(reinterpret_cast<float4*>(GA + (long long)i2 * C + c),
                                    make_float4(g[0] * w, g[1] * w, g[2] * w, g[3] * w));
                        gu = fmaf(g[3], x0.w - x2.w, fmaf(g[2], x0.z - x2.z,
                                                     fmaf(g[1], x0.y - x2.y, fmaf(g[0], x0.x - x2.x, gu))));
                        gv = fmaf(g[3], x1.w - x2.w, fmaf(g[2], x1.z - x2.z,
                                                     fmaf(g[1], x1.y - x2.y, fmaf(g[0], x1.x - x2.x, gv))));
                    }
                } else {
                    for (int c = q; c < C; c += LANES) {
                        const float g = aa_bwd_channel_g(at, grad, C, pix, c);
                        const float x0 = A[(long long)i0 * C + c], x1 = A[(long long)i1 * C + c],
                                    x2 = A[(long long)i2 * C + c];
                        atomicAdd(GA + (long long)i0 * C + c, g * u);
                        atomicAdd(GA + (long long)i1 * C + c, g * v);
                        atomicAdd(GA + (long long)i2 * C + c, g * w);
                        gu = fmaf(g, x0 - x2, gu);
                        gv = fmaf(g, x1 - x2, gv);
                    }
                }
            }
        }
#pragma unroll
        for (int off = 1; off < LANES; off <<= 1) {
            gu += __shfl_xor_sync(0xffffffffu, gu, off);
            gv += __shfl_xor_sync(0xffffffffu, gv, off);
        }
        if (active && t >= 0 && q == 0) {
            const drp_batch_item& it = *itp;
            const int W = it.width, H = it.height;
            const int py = pix / W, px = pix - py * W;
            const float X = fmaf((float)(2 * px + 1), __frcp_rn((float)W), -1.0f);
            const float Y = fmaf((float)(2 * py + 1), __frcp_rn((float)H), -1.0f);
            const float4* P = reinterpret_cast<const float4*>(a.pos) + it.pos_offset;
            float4* GP = reinterpret_cast<float4*>(a.grad_pos) + it.pos_offset;
            float4 g3[3];
            uv_grad_fast(P[i0], P[i1], P[i2], X, Y, gu, gv, g3);
            atomic_add4(GP + i0, make_float4(g3[0].x, g3[0].y, 0.f, g3[0].w));
            atomic_add4(GP + i1, make_float4(g3[1].x, g3[1].y, 0.f, g3[1].w));
            atomic_add4(GP + i2, make_float4(g3[2].x, g3[2].y, 0.f, g3[2].w));
        }
    }
}

// One resident wave of the listed-pixel kernel (its CTAs per SM from the
// occupancy query, cached per instantiation), capped by the pixel blocks.
template <int KIND>
static long long list_kernel_grid(long long pix_blocks) {
    static std::atomic<int> per_sm{0};
    int per = per_sm.load(std::memory_order_relaxed);
    if (per == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, batch_aa_bwd_kernel<KIND, kListLanes>, 256, 0);
        per = per > 0 ? per : 1;
        per_sm.store(per, std::memory_order_relaxed);
    }
    const int sms = drp_current_sm_count();
    const long long grid = (long long)(sms > 0 ? sms : 1) * per;
    return pix_blocks < grid ? pix_blocks : grid;
}

// Fused backward of one pixel: antialias colour gradient -> interpolation
// backward (attribute gradients, d/du, d/dv) -> rasterisation backward
// (vertex gradients).  Warps never straddle items (256-pixel blocks).
__global__ void __launch_bounds__(256, 4) batch_bwd_kernel(BatchArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    const int2 blk = a.pix_blocks[blockIdx.x];
    const drp_batch_item& it = a.items[blk.x];
    const int pix = blk.y * 256 + threadIdx.x;
    const int W = it.width, H = it.height, C = it.channels;
    const bool in = pix < W * H;
    const float4* R = reinterpret_cast<const float4*>(a.rast) + it.pixel_offset;
    const float* Cc = a.color + it.image_offset;
    const float* Gd = a.grad_out + it.image_offset;
    const float4* P = reinterpret_cast<const float4*>(a.pos) + it.pos_offset;
    float4* GP = reinterpret_cast<float4*>(a.grad_pos) + it.pos_offset;
    const int* tri = a.tri + 3 * (long long)it.tri_first;
    const float* A = a.attr + it.attr_offset;
    float* GA = a.grad_attr + it.attr_offset;
    const float4* rec = a.aa_rec + it.prim_offset * 2;

    // incoming gradients are multiplied by gsc as they are read (a fused
    // loss's upstream gradient; exactly 1 otherwise)
    const float gsc = a.grad_scale ? *a.grad_scale : 1.0f;
    AATerms at;
    at.any = false;
    int t = -1, i0 = 0, i1 = 0, i2 = 0;
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    // With the forward's antialias state, the pixels a blend touches belong
    // to batch_aa_bwd_kernel (their whole backward) and are skipped here; the
    // other pixels have no antialias terms.  Without it the terms are
    // evaluated here for every pixel.
    const bool flagged = in && a.aa_flags && a.aa_flags[it.pixel_offset + pix];
    if (in && !flagged) {
        if (!a.aa_flags) aa_bwd_terms(R, Cc, Gd, rec, it.tri_count, W, H, C, P, tri, GP, 1.0f, pix, at, gsc);
        r = R[pix];
        t = checked_tri(r.w, tri, it.tri_count, it.num_vertices, i0, i1, i2);
    }
    const Seg seg = seg_setup(t >= 0 ? (long long)t : (long long)(-1 - lane_id()));
    const float u = r.x, v = r.y, w = 1.0f - u - v;
    float gu = 0.f, gv = 0.f;
    const bool vec = (C & 3) == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(GA) |
                                       reinterpret_cast<uintptr_t>(Gd)) & 15) == 0;
    // Channel groups of 4: the next group's loads are issued before this
    // group's reduction and atomics, which would otherwise hold them back.
    float g[4], x0[4], x1[4], x2[4];
    auto load_group = [&](int c0) {
        if (vec) {
            const float4 gq = __ldg(reinterpret_cast<const float4*>(Gd + (long long)pix * C + c0));
            const float4 q0 = __ldg(reinterpret_cast<const float4*>(A + (long long)i0 * C + c0));
            const float4 q1 = __ldg(reinterpret_cast<const float4*>(A + (long long)i1 * C + c0));
            const float4 q2 = __ldg(reinterpret_cast<const float4*>(A + (long long)i2 * C + c0));
            g[0] = gq.x * gsc; g[1] = gq.y * gsc; g[2] = gq.z * gsc; g[3] = gq.w * gsc;
            x0[0] = q0.x; x0[1] = q0.y; x0[2] = q0.z; x0[3] = q0.w;
            x1[0] = q1.x; x1[1] = q1.y; x1[2] = q1.z; x1[3] = q1.w;
            x2[0] = q2.x; x2[1] = q2.y; x2[2] = q2.z; x2[3] = q2.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c = c0 + k < C ? c0 + k : C - 1;
                g[k] = c0 + k < C ? Gd[(long long)pix * C + c] * gsc : 0.f;
                x0[k] = A[(long long)i0 * C + c];
                x1[k] = A[(long long)i1 * C + c];
                x2[k] = A[(long long)i2 * C + c];
            }
        }
    };
    if (t >= 0) load_group(0);
    for (int c0 = 0; c0 < C; c0 += 4) {
        float val[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) val[k] = 0.f;
        if (t >= 0) {
            if (at.any) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (c0 + k < C) g[k] = aa_bwd_channel(at, Gd, C, pix, c0 + k, gsc);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                val[k] = g[k] * u;
                val[4 + k] = g[k] * v;
                val[8 + k] = g[k] * w;
                gu = fmaf(g[k], x0[k] - x2[k], gu);
                gv = fmaf(g[k], x1[k] - x2[k], gv);
            }
            if (c0 + 4 < C) load_group(c0 + 4);
        }
        seg_reduce<12>(seg, val);
        if (t >= 0 && seg.head) {
            if (vec) {
                atomic_add4(reinterpret_cast<float4*>(GA + (long long)i0 * C + c0),
                            make_float4(val[0], val[1], val[2], val[3]));
                atomic_add4(reinterpret_cast<float4*>(GA + (long long)i1 * C + c0),
                            make_float4(val[4], val[5], val[6], val[7]));
                atomic_add4(reinterpret_cast<float4*>(GA + (long long)i2 * C + c0),
                            make_float4(val[8], val[9], val[10], val[11]));
            } else {
                for (int k = 0; k < 4 && c0 + k < C; ++k) {
                    atomicAdd(GA + (long long)i0 * C + c0 + k, val[k]);
                    atomicAdd(GA + (long long)i1 * C + c0 + k, val[4 + k]);
                    atomicAdd(GA + (long long)i2 * C + c0 + k, val[8 + k]);
                }
            }
        }
    }
    // u and v do not depend on clip z, so each vertex gradient is (x, y, 0, w):
    // nine values to reduce
    float pv[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) pv[k] = 0.f;
    if (t >= 0) {
        const int py = pix / W, px = pix - py * W;
        const float X = fmaf((float)(2 * px + 1), __frcp_rn((float)W), -1.0f);
        const float Y = fmaf((float)(2 * py + 1), __frcp_rn((float)H), -1.0f);
        float4 g3[3];
        uv_grad_fast(P[i0], P[i1], P[i2], X, Y, gu, gv, g3);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            pv[3 * k] = g3[k].x;
            pv[3 * k + 1] = g3[k].y;
            pv[3 * k + 2] = g3[k].w;
        }
    }
    seg_reduce<9>(seg, pv);
    if (t >= 0 && seg.head) {
        atomic_add4(GP + i0, make_float4(pv[0], pv[1], 0.f, pv[2]));
        atomic_add4(GP + i1, make_float4(pv[3], pv[4], 0.f, pv[5]));
        atomic_add4(GP + i2, make_float4(pv[6], pv[7], 0.f, pv[8]));
    }
}

// Interpolated channels [c0, c0 + 4) of a pixel from its rast row and vertex
// indices (t < 0: background), as BatchEmit writes them; channels past C are 0.
// x0..x2 get the three vertices' values (0 for background).  VEC: C % 4 == 0
// and 16-byte aligned attributes.
template <bool VEC>
__device__ __forceinline__ void lerp_group(const float* A, int C, int c0, int t, int i0, int i1, int i2, float u,
                                           float v, float (&x0)[4], float (&x1)[4], float (&x2)[4], float (&col)[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) x0[k] = x1[k] = x2[k] = col[k] = 0.f;
    if (t < 0) return;
    if (VEC) {
        const float4 q0 = __ldg(reinterpret_cast<const float4*>(A + (long long)i0 * C + c0));
        const float4 q1 = __ldg(reinterpret_cast<const float4*>(A + (long long)i1 * C + c0));
        const float4 q2 = __ldg(reinterpret_cast<const float4*>(A + (long long)i2 * C + c0));
        x0[0] = q0.x; x0[1] = q0.y; x0[2] = q0.z; x0[3] = q0.w;
        x1[0] = q1.x; x1[1] = q1.y; x1[2] = q1.z; x1[3] = q1.w;
        x2[0] = q2.x; x2[1] = q2.y; x2[2] = q2.z; x2[3] = q2.w;
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (c0 + k < C) {
                x0[k] = A[(long long)i0 * C + c0 + k];
                x1[k] = A[(long long)i1 * C + c0 + k];
                x2[k] = A[(long long)i2 * C + c0 + k];
            }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) col[k] = fmaf(x0[k] - x2[k], u, fmaf(x1[k] - x2[k], v, x2[k]));
}

// l1_sign in three instructions (setp.ne is false for NaN, as both compares are).
__device__ __forceinline__ float l1_sign_fast(float d, float scale) {
    float g;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.f32 p, %1, 0f00000000;\n\tselp.f32 %0, %2, 0f00000000, p;\n\t}"
        : "=f"(g)
        : "f"(d), "f"(__uint_as_float((__float_as_uint(d) & 0x80000000u) ^ __float_as_uint(scale))));
    return g;
}

// The same four written back (load_channels).
template <bool VEC>
__device__ __forceinline__ void store4(float* p, int n, const float (&x)[4]) {
    if (VEC) {
        *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < n) p[k] = x[k];
    }
}

// Antialias + L1 loss with the loss's gradient formed in the same pass, for
// large launches (fit_words_bytes; drp_batch_fit_l1,
// drp_batch_forward_l1_grad).  Every pixel: its colour, interpolated again
// from its rast row (the attribute rows are needed for the backward anyway, so
// no colour image is written and read back), the blend, the output and the
// |error| sum.  Then, for the pixels no blending pair touches (the listed ones
// belong to batch_aa_bwd_kernel, which forms the sign from the output
// and the target), the pixel's whole backward with g = sign(out - target) *
// scale, as batch_aa_l1_grad_kernel forms it.
//
// A warp first finds the pairs that may blend and evaluates them together
// (fit_pairs), then walks its rows down, one column per lane, and keeps the
// sums of the triangle its column is in as registers (eight channels x three
// vertices and the three positions): a triangle several pixels tall costs one
// fused multiply-add per value and pixel, and a row of floats in shared memory
// only where a column leaves it.  32 such rows are then added by columns and
// go out with one vector atomic per run of rows of one triangle (fit_drain).
// Rast rows and target come by asynchronous copies two rows ahead.
//
// What bounds it: issue and the latency of the gathers at 16 warps per SM.
// One thread per pixel with segmented shuffles took 1270 warp instructions
// per 32 pixels on 64 views of 512 x 512 x 8 channels, most of them predicated
// shuffle steps and pair evaluation for a lane or two at a time; this takes
// about 500, and the pass 516 instead of 951 us; on one 1024 x 1024 view 65
// instead of 77 us.
// Floats per shared row: 24 attribute sums (per four channels three vertices),
// three position sums (x, y, 0, w), the vertex indices; eight lanes' float4
// stores cover the banks.
constexpr int kFitRow = 44;
constexpr int kFitStages = 3;  // rows of a walk in flight or in use

// One warp's shared memory: the pair terms (PairShared) first, then the walk.
struct FitWalkShared {
    float rows[32][kFitRow];
    float4 rast[kFitStages][32];       // the walk's rows: rast and
    float4 target[kFitStages][2][32];  // target (groups of four channels)
};
template <int ROWS>
union FitShared {
    PairShared<ROWS> p;
    FitWalkShared w;
};

// Adds the first n rows of sh.rows into the gradients: NG groups of four
// channels from c0 and, with POS, the clip positions.  Lane (r, q) adds quad q
// of the r-th part of the rows; where a run of rows of one triangle (or the
// part) ends, one vector atomic adds its four sums.
template <int NG, bool POS, bool VEC>
__device__ __forceinline__ void fit_drain(const BatchArgs& a, const drp_batch_item& it, FitWalkShared& sh, int n,
                                          int c0) {
    constexpr int Q = 3 * NG + (POS ? 3 : 0), PARTS = 32 / Q, LEN = (32 + PARTS - 1) / PARTS;
    const int lane = threadIdx.x & 31, C = it.channels;
    __syncwarp();
    int4 id = make_int4(-1, -1, -1, 0);
    if (lane < n) id = *reinterpret_cast<const int4*>(&sh.rows[lane][36]);
    const int nx = __shfl_down_sync(0xffffffffu, id.x, 1), ny = __shfl_down_sync(0xffffffffu, id.y, 1),
              nz = __shfl_down_sync(0xffffffffu, id.z, 1);
    const unsigned ends = __ballot_sync(0xffffffffu, lane == 31 || nx != id.x || ny != id.y || nz != id.z);
    const int rq = lane / Q, cq = lane - rq * Q, first = rq * LEN, len = min(n - first, LEN);
    if (rq < PARTS && len > 0) {
        const unsigned my_ends = (ends >> first) | (1u << (len - 1));
        const bool attr_q = cq < 3 * NG;
        const int slot = cq % 3, cg = c0 + 4 * (cq / 3);
        float* base = attr_q ? a.grad_attr + it.attr_offset + cg : a.grad_pos + 4 * it.pos_offset;
        const int stride = attr_q ? C : 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < LEN; ++k) {
            if (k >= len) break;
            const float* row = sh.rows[first + k];
            const float4 x = *reinterpret_cast<const float4*>(row + 4 * cq);
            acc.x += x.x;
            acc.y += x.y;
            acc.z += x.z;
            acc.w += x.w;
            if ((my_ends >> k) & 1u) {
                float* d = base + (long long)__float_as_int(row[36 + slot]) * stride;
                if (VEC || !attr_q) {
                    atomic_add4(reinterpret_cast<float4*>(d), acc);
                } else {
                    atomicAdd(d, acc.x);
                    if (cg + 1 < C) atomicAdd(d + 1, acc.y);
                    if (cg + 2 < C) atomicAdd(d + 2, acc.z);
                    if (cg + 3 < C) atomicAdd(d + 3, acc.w);
                }
                acc = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    __syncwarp();
}

// What a pixel of the warp's rows is, one bit per row and lane: on a triangle
// and in no blending pair (live: its backward is done here), written here (not
// blended into), and in the list of batch_aa_bwd_kernel.
struct FitClass {
    unsigned live, plain, listed;
};

// Pair terms of the rows [y0, y1) (at most ROWS) x columns [x0, x0 + 32) by one
// warp (warp_pairs, from the words the fine raster wrote), and with them
// everything of the pixels a pair blends into: their output and |error|
// (returned, per lane).  The blended pixels are done one lane per (pixel, group
// of four channels), and the listed ones take their places in the list with
// one atomic.  LOSS = false (rendering): the blended pixels' output only, no
// list and no error.
template <bool VEC, int ROWS, bool LOSS>
__device__ __noinline__ float fit_pairs(const BatchArgs& a, const drp_batch_item& it, PairShared<ROWS>& sh,
                                        int x0, int y0, int y1, FitClass& cl) {
    const int lane = threadIdx.x & 31, x = x0 + lane;
    const int W = it.width, H = it.height, C = it.channels;
    const bool in = x < W;
    const float4* R = reinterpret_cast<const float4*>(a.rast) + it.pixel_offset;
    const uint32_t* Wd = a.aa_words + it.pixel_offset;
    const int* tri = a.tri + 3 * (long long)it.tri_first;
    const float* A = a.attr + it.attr_offset;
    const int p0 = y0 * W + x;
    uint32_t w[ROWS + 2], side[ROWS];  // rows y0 - 1 .. y1
#pragma unroll
    for (int r = 0; r < ROWS + 2; ++r) {
        const int y = y0 - 1 + r;
        w[r] = in && y >= 0 && y < H && y <= y1 ? Wd[p0 + (r - 1) * W] : 0u;
    }
    const bool edge = (lane == 0 && x > 0) || (lane == 31 && x + 1 < W);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) side[r] = y0 + r < y1 && edge ? Wd[p0 + r * W + (lane == 0 ? -1 : 1)] : 0u;
    cl.live = cl.plain = cl.listed = 0u;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (!in || y0 + r >= y1) continue;
        cl.plain |= 1u << r;
        if (w[r + 1] & ~kPixSil) cl.live |= 1u << r;
    }
    float sum = 0.f, low = 0.f;
    unsigned listed, blended;
    const auto depth = [&](int pix, int, int) { return reinterpret_cast<const float*>(R + pix)[2]; };
    if (warp_pairs<ROWS>(depth, a.aa_rec + it.prim_offset * 2, W, H, x0, y0, y1, w, side, sh, listed, blended)) {
        if (LOSS) cl.listed = listed;
        cl.live &= ~cl.listed;
        cl.plain &= ~blended;
        // listed pixels
        if (LOSS) {
            const int lend = warp_prefix(__popc(cl.listed));
            unsigned base = 0u;
            if (lane == 31 && lend) base = atomicAdd(a.aa_count, (unsigned)lend);
            base = __shfl_sync(0xffffffffu, base, 31) + (unsigned)(lend - __popc(cl.listed));
            for (unsigned m = cl.listed; m; m &= m - 1)
                a.aa_list[base++] = (int)(it.pixel_offset + p0 + (__ffs(m) - 1) * W);
        }
        // blended pixels
        const int bend = warp_prefix(__popc(blended)), nb = __shfl_sync(0xffffffffu, bend, 31);
        {
            int e = bend - __popc(blended);
            for (unsigned m = blended; m; m &= m - 1) sh.blend[e++] = (unsigned short)(lane | ((__ffs(m) - 1) << 5));
        }
        __syncwarp();
        const int per = (C + 3) >> 2, tasks = nb * per;
#pragma unroll 1
        for (int k = lane; k < tasks; k += 32) {
            const int e = k / per, cg = 4 * (k - e * per);
            const int l = sh.blend[e] & 31, r = sh.blend[e] >> 5;
            const int p = (y0 + r) * W + x0 + l;
            int slots = (int)(sh.flags[r][l] >> 4);
            const long long prow = it.image_offset + (long long)p * C + cg;
            float tg[4], y[3][4], base4[4], sv[4], val[4];
            if (LOSS) load_channels<VEC>(a.target + prow, C - cg, tg);
            // the pixel and its sources in slot order (one as a rule): each
            // source's gathers are issued beside the ones before it
            auto vertices = [&](int sp, uint32_t word, float4& rp, int& t, int& j0, int& j1, int& j2) {
                rp = R[sp];
                t = (int)(word & ~kPixSil) - 1;
                j0 = j1 = j2 = 0;
                if (t >= 0) {
                    j0 = tri[3 * (long long)t];
                    j1 = tri[3 * (long long)t + 1];
                    j2 = tri[3 * (long long)t + 2];
                }
            };
            float4 rp, rs;
            int t, j0, j1, j2, ts, k0, k1, k2;
            vertices(p, sh.words[r + 1][l + 1], rp, t, j0, j1, j2);
            int q = __ffs(slots) - 1;
            auto source = [&]() {
                const int dx = q == 0 ? -1 : (q == 1 ? 1 : 0), dy = q == 2 ? -1 : (q == 3 ? 1 : 0);
                vertices(p + dx + dy * W, sh.words[r + 1 + dy][l + 1 + dx], rs, ts, k0, k1, k2);
            };
            source();
            lerp_group<VEC>(A, C, cg, t, j0, j1, j2, rp.x, rp.y, y[0], y[1], y[2], base4);
#pragma unroll
            for (int c = 0; c < 4; ++c) val[c] = base4[c];
            for (;;) {
                lerp_group<VEC>(A, C, cg, ts, k0, k1, k2, rs.x, rs.y, y[0], y[1], y[2], sv);
                const float wq = sh.wt[r][l][q];
#pragma unroll
                for (int c = 0; c < 4; ++c) val[c] = fmaf(wq, sv[c] - base4[c], val[c]);
                slots &= slots - 1;
                if (!slots) break;
                q = __ffs(slots) - 1;
                source();
            }
            store4<VEC>(a.out + prow, C - cg, val);
            if (LOSS) {
                float s4 = 0.f;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (VEC || cg + c < C) s4 += fabsf(val[c] - tg[c]);
                kahan_add(sum, low, s4);
            }
        }
    }
    if (C > 32) cl.live = 0u;
    return sum;
}

// Four channels (those below n) as two pairs.
template <bool VEC>
__device__ __forceinline__ ulonglong2 load_pairs(const float* p, int n) {
    if constexpr (VEC) {
        return __ldg(reinterpret_cast<const ulonglong2*>(p));
    } else {
        float x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = k < n ? __ldg(p + k) : 0.f;
        return make_ulonglong2(pack2(x[0], x[1]), pack2(x[2], x[3]));
    }
}

// The rows [y0, y1) x columns [x0, x0 + 32) of an item of 4 NG channels with
// 16-byte aligned rows (VEC), or of up to 4 NG channels, by one warp; returns
// the lane's |error| sum.  Pairs of channels share instructions (fma2).
template <int NG, bool VEC>
__device__ __forceinline__ float fit_walk(const BatchArgs& a, const drp_batch_item& it, FitWalkShared& sh, int x0,
                                          int y0, int y1, const FitClass& cl) {
    const int C = VEC ? 4 * NG : it.channels;
    const int lane = threadIdx.x & 31, x = x0 + lane;
    const int W = it.width;
    const bool in = x < W;
    const float4* R = reinterpret_cast<const float4*>(a.rast) + it.pixel_offset;
    const uint32_t* Wd = a.aa_words + it.pixel_offset;
    const int* tri = a.tri + 3 * (long long)it.tri_first;
    const float* A = a.attr + it.attr_offset;
    const long long image_offset = it.image_offset;  // the stores below could alias it
    const float4* P = reinterpret_cast<const float4*>(a.pos) + it.pos_offset;
    const float X = fmaf((float)(2 * x + 1), __frcp_rn((float)W), -1.0f), rh = __frcp_rn((float)it.height);
    const f32x2 minus1 = pack2(-1.0f, -1.0f);
    float s = 0.f, low = 0.f;
    int n = 0;
    // the column's triangle: sums (vertex i, channels 2 k, 2 k + 1), position sums, vertices
    f32x2 acc[3][2 * NG];
    float pv[9];
    int cur = -1, j0 = 0, j1 = 0, j2 = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 2 * NG; ++k) acc[i][k] = 0ull;
#pragma unroll
    for (int k = 0; k < 9; ++k) pv[k] = 0.f;
    auto leave = [&](int e) {  // the column's sums as row e
        f32x2* d = reinterpret_cast<f32x2*>(sh.rows[e]);
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int i = 0; i < 3; ++i)
                *reinterpret_cast<ulonglong2*>(d + 6 * g + 2 * i) = make_ulonglong2(acc[i][2 * g], acc[i][2 * g + 1]);
#pragma unroll
        for (int i = 0; i < 3; ++i)
            *reinterpret_cast<float4*>(d + 6 * NG + 2 * i) =
                make_float4(pv[3 * i], pv[3 * i + 1], 0.f, pv[3 * i + 2]);
        *reinterpret_cast<int4*>(d + 18) = make_int4(j0, j1, j2, 0);
    };

    // Rast rows and target arrive in shared memory two rows ahead of their use
    // (asynchronous copies: they hold no registers), words too, vertex indices one.
    int pix = y0 * W + x;
    auto request = [&](int y) {
        if (in && y < y1) {
            const int st = (y - y0) % kFitStages, p = y * W + x;
            cp_async<16>(&sh.rast[st][lane], R + p);
            const float* tg = a.target + image_offset + (long long)p * C;
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                float* d = reinterpret_cast<float*>(&sh.target[st][g][lane]);
                if (VEC) {
                    cp_async<16>(d, tg + 4 * g);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (4 * g + k < C) cp_async<4>(d + k, tg + 4 * g + k);
                }
            }
        }
        cp_async_commit();
    };
    if (!VEC) {  // channels past the last stay zero
#pragma unroll
        for (int k = 0; k < kFitStages; ++k)
#pragma unroll
            for (int c = 0; c < 4 * NG; ++c)
                if (c >= C) reinterpret_cast<float*>(&sh.target[k][c >> 2][lane])[c & 3] = 0.f;
    }
    request(y0);
    request(y0 + 1);
    int t = -1, t_n = -1, i0 = 0, i1 = 0, i2 = 0;
    if (in) {
        t = (int)(Wd[pix] & ~kPixSil) - 1;
        if (y0 + 1 < y1) t_n = (int)(Wd[pix + W] & ~kPixSil) - 1;
    }
    if (t >= 0) {
        i0 = tri[3 * (long long)t];
        i1 = tri[3 * (long long)t + 1];
        i2 = tri[3 * (long long)t + 2];
    }
    int st = 0;
#pragma unroll 1
    for (int yy = y0; yy < y1; ++yy) {
        const unsigned bit = 1u << (yy - y0);
        request(yy + 2);
        int t_nn = -1, n0 = 0, n1 = 0, n2 = 0;
        if (in && yy + 2 < y1) t_nn = (int)(Wd[pix + 2 * W] & ~kPixSil) - 1;
        if (t_n >= 0) {
            n0 = tri[3 * (long long)t_n];
            n1 = tri[3 * (long long)t_n + 1];
            n2 = tri[3 * (long long)t_n + 2];
        }
        const bool live = cl.live & bit;

        // a column that enters another triangle leaves its sums behind
        const bool enter = live && t != cur;
        const unsigned fm = __ballot_sync(0xffffffffu, enter && cur >= 0);
        if (fm) {
            if (n + __popc(fm) > 32) {
                fit_drain<NG, true, VEC>(a, it, sh, n, 0);
                n = 0;
            }
            if (enter && cur >= 0) leave(n + __popc(fm & ((1u << lane) - 1u)));
            n += __popc(fm);
        }
        if (enter) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int k = 0; k < 2 * NG; ++k) acc[i][k] = 0ull;
#pragma unroll
            for (int k = 0; k < 9; ++k) pv[k] = 0.f;
            cur = t;
            j0 = i0;
            j1 = i1;
            j2 = i2;
        }

        cp_async_wait<2>();  // row yy (this lane's part)
        const float4 r = in ? sh.rast[st][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        // pixels that add nothing take zero barycentrics
        const float bu = live ? r.x : 0.f, bv = live ? r.y : 0.f, bw = live ? 1.0f - r.x - r.y : 0.f;
        const f32x2 uu = pack2(r.x, r.x), vv = pack2(r.y, r.y);
        const f32x2 bb[3] = {pack2(bu, bu), pack2(bv, bv), pack2(bw, bw)};
        float gu = 0.f, gv = 0.f, sr = 0.f;
        const long long row = image_offset + (long long)pix * C;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            ulonglong2 x0v = make_ulonglong2(0ull, 0ull), x1v = x0v, x2v = x0v, tv = x0v;
            if (t >= 0) {
                x0v = load_pairs<VEC>(A + (long long)i0 * C + 4 * g, C - 4 * g);
                x1v = load_pairs<VEC>(A + (long long)i1 * C + 4 * g, C - 4 * g);
                x2v = load_pairs<VEC>(A + (long long)i2 * C + 4 * g, C - 4 * g);
            }
            if (in) tv = *reinterpret_cast<const ulonglong2*>(&sh.target[st][g][lane]);
            f32x2 val[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const f32x2 a0 = k ? x0v.y : x0v.x, a1 = k ? x1v.y : x1v.x, a2 = k ? x2v.y : x2v.x;
                const f32x2 d0 = fma2(a2, minus1, a0), d1 = fma2(a2, minus1, a1);
                val[k] = fma2(d0, uu, fma2(d1, vv, a2));
                const f32x2 d = fma2(k ? tv.y : tv.x, minus1, val[k]);
                sr += fabsf(lo2(d));
                sr += fabsf(hi2(d));
                const float g0 = l1_sign_fast(lo2(d), a.l1_scale), g1 = l1_sign_fast(hi2(d), a.l1_scale);
                gu = fmaf(g1, hi2(d0), fmaf(g0, lo2(d0), gu));
                gv = fmaf(g1, hi2(d1), fmaf(g0, lo2(d1), gv));
                const f32x2 gg = pack2(g0, g1);
#pragma unroll
                for (int i = 0; i < 3; ++i) acc[i][2 * g + k] = fma2(gg, bb[i], acc[i][2 * g + k]);
            }
            const float v4[4] = {lo2(val[0]), hi2(val[0]), lo2(val[1]), hi2(val[1])};
            if (cl.plain & bit) store4<VEC>(a.out + row + 4 * g, C - 4 * g, v4);
            if ((cl.listed & bit) && !a.emit_color)  // for the listed pixels' kernel
                store4<VEC>(a.color + row + 4 * g, C - 4 * g, v4);
        }
        if (cl.plain & bit) kahan_add(s, low, sr);
        if (live) {
            float4 g3[3];
            uv_grad_fast(P[i0], P[i1], P[i2], X, fmaf((float)(2 * yy + 1), rh, -1.0f), gu, gv, g3);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                pv[3 * i] += g3[i].x;
                pv[3 * i + 1] += g3[i].y;
                pv[3 * i + 2] += g3[i].w;
            }
        }
        t = t_n;
        t_n = t_nn;
        i0 = n0;
        i1 = n1;
        i2 = n2;
        pix += W;
        st = st + 1 == kFitStages ? 0 : st + 1;
    }
    // what the columns still hold
    const unsigned fm = __ballot_sync(0xffffffffu, cur >= 0);
    if (n + __popc(fm) > 32) {
        fit_drain<NG, true, VEC>(a, it, sh, n, 0);
        n = 0;
    }
    if (cur >= 0) leave(n + __popc(fm & ((1u << lane) - 1u)));
    n += __popc(fm);
    if (n) fit_drain<NG, true, VEC>(a, it, sh, n, 0);
    return s;
}

// The same for any channel count and alignment: each pixel's values are the
// row (no sums held over rows: the registers hold eight channels at a time),
// the 32 rows of a row of pixels are added at once.
template <bool VEC>
__device__ __forceinline__ float fit_rows(const BatchArgs& a, const drp_batch_item& it, FitWalkShared& sh, int x0,
                                          int y0, int y1, const FitClass& cl) {
    const int lane = threadIdx.x & 31, x = x0 + lane;
    const int W = it.width, C = it.channels;
    const bool in = x < W;
    const float4* R = reinterpret_cast<const float4*>(a.rast) + it.pixel_offset;
    const uint32_t* Wd = a.aa_words + it.pixel_offset;
    const int* tri = a.tri + 3 * (long long)it.tri_first;
    const float* A = a.attr + it.attr_offset;
    const long long image_offset = it.image_offset;
    const float X = fmaf((float)(2 * x + 1), __frcp_rn((float)W), -1.0f), rh = __frcp_rn((float)it.height);
    const float sc = a.l1_scale;
    float s = 0.f, low = 0.f;
    int pix = y0 * W + x;
#pragma unroll 1
    for (int yy = y0; yy < y1; ++yy, pix += W) {
        const unsigned bit = 1u << (yy - y0);
        const long long row = image_offset + (long long)pix * C;
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        float tv[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        int t = -1, i0 = 0, i1 = 0, i2 = 0;
        if (in) {
            t = (int)(Wd[pix] & ~kPixSil) - 1;
            r = R[pix];
            load_channels<VEC>(a.target + row, C, tv[0]);
            if (C > 4) load_channels<VEC>(a.target + row + 4, C - 4, tv[1]);
            if (t >= 0) {
                i0 = tri[3 * (long long)t];
                i1 = tri[3 * (long long)t + 1];
                i2 = tri[3 * (long long)t + 2];
            }
        }
        const bool plain = cl.plain & bit, live = cl.live & bit;
        const bool keep_color = (cl.listed & bit) && !a.emit_color;  // for the listed pixels' kernel
        const unsigned live_mask = __ballot_sync(0xffffffffu, live);
        const int n = __popc(live_mask);
        float* rw = sh.rows[__popc(live_mask & ((1u << lane) - 1u))];
        if (live) *reinterpret_cast<int4*>(rw + 36) = make_int4(i0, i1, i2, 0);
        const float u = r.x, v = r.y, w = 1.0f - u - v;
        float gu = 0.f, gv = 0.f, sr = 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < C; c0 += 8) {
            const int ng = C - c0 > 4 ? 2 : 1;
            const bool last = c0 + 8 >= C;
#pragma unroll
            for (int gi = 0; gi < 2; ++gi) {
                if (gi >= ng) break;
                const int cg = c0 + 4 * gi;
                float q0[4], q1[4], q2[4], val[4], g[4];
                lerp_group<VEC>(A, C, cg, t, i0, i1, i2, u, v, q0, q1, q2, val);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float d = plain && (VEC || cg + k < C) ? val[k] - tv[gi][k] : 0.f;
                    sr += fabsf(d);
                    g[k] = l1_sign_fast(d, sc);
                }
                if (plain) store4<VEC>(a.out + row + cg, C - cg, val);
                if (keep_color) store4<VEC>(a.color + row + cg, C - cg, val);
                if (in && cg + 8 < C) load_channels<VEC>(a.target + row + cg + 8, C - cg - 8, tv[gi]);
                if (live) {
                    float4* d = reinterpret_cast<float4*>(rw + 12 * gi);
                    d[0] = make_float4(g[0] * u, g[1] * u, g[2] * u, g[3] * u);
                    d[1] = make_float4(g[0] * v, g[1] * v, g[2] * v, g[3] * v);
                    d[2] = make_float4(g[0] * w, g[1] * w, g[2] * w, g[3] * w);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        gu = fmaf(g[k], q0[k] - q2[k], gu);
                        gv = fmaf(g[k], q1[k] - q2[k], gv);
                    }
                }
            }
            if (last && live) {
                const float4* P = reinterpret_cast<const float4*>(a.pos) + it.pos_offset;
                float4 g3[3];
                uv_grad_fast(P[i0], P[i1], P[i2], X, fmaf((float)(2 * yy + 1), rh, -1.0f), gu, gv, g3);
                float4* d = reinterpret_cast<float4*>(rw + 12 * ng);
#pragma unroll
                for (int i = 0; i < 3; ++i) d[i] = make_float4(g3[i].x, g3[i].y, 0.f, g3[i].w);
            }
            if (!n) continue;
            if (last && ng == 2) fit_drain<2, true, VEC>(a, it, sh, n, c0);
            else if (last) fit_drain<1, true, VEC>(a, it, sh, n, c0);
            else fit_drain<2, false, VEC>(a, it, sh, n, c0);
        }
        kahan_add(s, low, sr);
    }
    return s;
}

// Rendering: blends the pixels that a pair touches into the image the fine
// raster wrote.  One warp per 32 x ROWS pixels, on its own: most warps read
// their words and are done.  What bounds it: the chain of dependent loads of
// the pairs that blend (rows per warp: kBlendTallPixels).  Against one thread
// per pixel testing the four pairs of its rast rows, with the colours kept
// apart from the images so that a pair reads unblended ones: 84 instead of
// 162 us for 5.8M pixels of ten meshes, and the fine raster, which then writes
// one image instead of two, 443 instead of 619 us.
constexpr int kBlendWarps = 4;
template <int ROWS>
__global__ void __launch_bounds__(32 * kBlendWarps) batch_blend_kernel(const __grid_constant__ BatchArgs a) {
    __shared__ PairShared<ROWS> sh[kBlendWarps];
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, per_tile = 16 / ROWS * fit_regions_per_tile(a.tile_log2);
    const long long unit = (long long)blockIdx.x * kBlendWarps + warp, tile_id = unit / per_tile;
    if (tile_id >= a.total_tiles) return;
    const drp_batch_item& it = a.items[find_item_by_tile(a.items, a.num_items, tile_id)];
    const int tile = (int)(tile_id - it.tile_offset);
    const int ty = tile / it.tiles_x, tx = tile - ty * it.tiles_x;
    if (!fit_region_owner(a.tile_log2, tx, ty)) return;
    const int y0 = (ty << a.tile_log2) + (int)(unit % per_tile) * ROWS, y1 = min(y0 + ROWS, it.height);
    if (y0 >= y1) return;
    const bool vec = (it.channels & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.attr + it.attr_offset) |
                                                 reinterpret_cast<uintptr_t>(a.out + it.image_offset)) & 15) == 0;
    FitClass cl;
    if (vec) fit_pairs<true, ROWS, false>(a, it, sh[warp], tx << a.tile_log2, y0, y1, cl);
    else fit_pairs<false, ROWS, false>(a, it, sh[warp], tx << a.tile_log2, y0, y1, cl);
}

// One region of 32 x 16 pixels per CTA: WARPS warps of 16 / WARPS rows.
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 16 / WARPS) batch_fit_kernel(const __grid_constant__ BatchArgs a) {
    constexpr int ROWS = 16 / WARPS;
    __shared__ __align__(16) FitShared<ROWS> sh[WARPS];
    __shared__ float warp_sum[WARPS];
    pdl_wait();
    pdl_launch_dependents();
    const int per_tile = fit_regions_per_tile(a.tile_log2);
    const long long tile_id = blockIdx.x / per_tile;
    const drp_batch_item& it = a.items[find_item_by_tile(a.items, a.num_items, tile_id)];
    const int tile = (int)(tile_id - it.tile_offset);
    const int ty = tile / it.tiles_x, tx = tile - ty * it.tiles_x;
    const bool owner = fit_region_owner(a.tile_log2, tx, ty);
    const int warp = threadIdx.x >> 5;
    const int x0 = tx << a.tile_log2;
    const int y0 = (ty << a.tile_log2) + (int)(blockIdx.x % per_tile) * 16 + ROWS * warp;
    const int y1 = min(y0 + ROWS, it.height);
    float s = 0.f;
    if (owner && y0 < y1) {
        const bool vec = (it.channels & 3) == 0 &&
                         ((reinterpret_cast<uintptr_t>(a.attr + it.attr_offset) |
                           reinterpret_cast<uintptr_t>(a.grad_attr + it.attr_offset) |
                           reinterpret_cast<uintptr_t>(a.target + it.image_offset) |
                           reinterpret_cast<uintptr_t>(a.out + it.image_offset) |
                           reinterpret_cast<uintptr_t>(a.color + it.image_offset)) & 15) == 0;
        FitClass cl;
        if (vec) s = fit_pairs<true, ROWS, true>(a, it, sh[warp].p, x0, y0, y1, cl);
        else s = fit_pairs<false, ROWS, true>(a, it, sh[warp].p, x0, y0, y1, cl);
        __syncwarp();  // the pair terms' shared memory becomes the walk's
        // walks hold the sums of four or eight channels; see fit_rows
        if (vec && it.channels == 8) s += fit_walk<2, true>(a, it, sh[warp].w, x0, y0, y1, cl);
        else if (vec && it.channels == 4) s += fit_walk<1, true>(a, it, sh[warp].w, x0, y0, y1, cl);
        else if (it.channels <= 4) s += fit_walk<1, false>(a, it, sh[warp].w, x0, y0, y1, cl);
        else if (it.channels <= 8) s += fit_walk<2, false>(a, it, sh[warp].w, x0, y0, y1, cl);
        else if (vec) s += fit_rows<true>(a, it, sh[warp].w, x0, y0, y1, cl);
        else s += fit_rows<false>(a, it, sh[warp].w, x0, y0, y1, cl);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) warp_sum[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = warp_sum[0];
#pragma unroll
        for (int k = 1; k < WARPS; ++k) sum += warp_sum[k];
        *fit_loss_slot(a, blockIdx.x) = sum;
        if (it.channels > 32) atomicOr(a.stats + 2, DRP_DEVERR_CHANNELS);
    }
}

// The backward of one pixel no blending pair touches, with the upstream
// gradient sign(out - target) * scale given by the sign masks (bit c:
// nonzero / positive): interpolation backward (attribute gradients) and
// rasterisation backward (vertex gradients), reduced over runs of one
// triangle in the warp and scattered with float4 atomics.  All 32 lanes call
// it (active = false for the others); a warp without an active lane on a
// triangle returns at once.
// r, t, i0..i2: the pixel's rast row, triangle (-1: none, or not active)
// and vertex indices, loaded by the caller before its antialias work.
__device__ __forceinline__ void pixel_backward_l1(const BatchArgs& a, const drp_batch_item& it, int pix, float4 r,
                                                  int t, int i0, int i1, int i2, unsigned nz, unsigned ps) {
    const int W = it.width, H = it.height, C = it.channels;
    const float* A = a.attr + it.attr_offset;
    float* GA = a.grad_attr + it.attr_offset;
    const float4* P = reinterpret_cast<const float4*>(a.pos) + it.pos_offset;
    float4* GP = reinterpret_cast<float4*>(a.grad_pos) + it.pos_offset;
    if (!__any_sync(0xffffffffu, t >= 0)) return;  // background or listed pixels only: nothing to add
    const Seg seg = seg_setup(t >= 0 ? (long long)t : (long long)(-1 - lane_id()));
    const float u = r.x, v = r.y, w = 1.0f - u - v;
    const float sc = a.l1_scale;
    float gu = 0.f, gv = 0.f;
    const bool vec = (C & 3) == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(GA)) & 15) == 0;
    for (int c0 = 0; c0 < C; c0 += 4) {
        float val[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) val[k] = 0.f;
        if (t >= 0) {
            float g[4], x0[4], x1[4], x2[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c = c0 + k;
                g[k] = (c < C && ((nz >> c) & 1u)) ? (((ps >> c) & 1u) ? sc : -sc) : 0.f;
            }
            if (vec) {
                const float4 q0 = __ldg(reinterpret_cast<const float4*>(A + (long long)i0 * C + c0));
                const float4 q1 = __ldg(reinterpret_cast<const float4*>(A + (long long)i1 * C + c0));
                const float4 q2 = __ldg(reinterpret_cast<const float4*>(A + (long long)i2 * C + c0));
                x0[0] = q0.x; x0[1] = q0.y; x0[2] = q0.z; x0[3] = q0.w;
                x1[0] = q1.x; x1[1] = q1.y; x1[2] = q1.z; x1[3] = q1.w;
                x2[0] = q2.x; x2[1] = q2.y; x2[2] = q2.z; x2[3] = q2.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int c = c0 + k < C ? c0 + k : C - 1;
                    x0[k] = A[(long long)i0 * C + c];
                    x1[k] = A[(long long)i1 * C + c];
                    x2[k] = A[(long long)i2 * C + c];
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                val[k] = g[k] * u;
                val[4 + k] = g[k] * v;
                val[8 + k] = g[k] * w;
                gu = fmaf(g[k], x0[k] - x2[k], gu);
                gv = fmaf(g[k], x1[k] - x2[k], gv);
            }
        }
        seg_reduce<12>(seg, val);
        if (t >= 0 && seg.head) {
            if (vec) {
                atomic_add4(reinterpret_cast<float4*>(GA + (long long)i0 * C + c0),
                            make_float4(val[0], val[1], val[2], val[3]));
                atomic_add4(reinterpret_cast<float4*>(GA + (long long)i1 * C + c0),
                            make_float4(val[4], val[5], val[6], val[7]));
                atomic_add4(reinterpret_cast<float4*>(GA + (long long)i2 * C + c0),
                            make_float4(val[8], val[9], val[10], val[11]));
            } else {
                for (int k = 0; k < 4 && c0 + k < C; ++k) {
                    atomicAdd(GA + (long long)i0 * C + c0 + k, val[k]);
                    atomicAdd(GA + (long long)i1 * C + c0 + k, val[4 + k]);
                    atomicAdd(GA + (long long)i2 * C + c0 + k, val[8 + k]);
                }
            }
        }
    }
    float pv[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) pv[k] = 0.f;
    if (t >= 0) {
        const int py = pix / W, px = pix - py * W;
        const float X = fmaf((float)(2 * px + 1), __frcp_rn((float)W), -1.0f);
        const float Y = fmaf((float)(2 * py + 1), __frcp_rn((float)H), -1.0f);
        float4 g3[3];
        uv_grad_fast(P[i0], P[i1], P[i2], X, Y, gu, gv, g3);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            pv[3 * k] = g3[k].x;
            pv[3 * k + 1] = g3[k].y;
            pv[3 * k + 2] = g3[k].w;
        }
    }
    seg_reduce<9>(seg, pv);
    if (t >= 0 && seg.head) {
        atomic_add4(GP + i0, make_float4(pv[0], pv[1], 0.f, pv[2]));
        atomic_add4(GP + i1, make_float4(pv[3], pv[4], 0.f, pv[5]));
        atomic_add4(GP + i2, make_float4(pv[6], pv[7], 0.f, pv[8]));
    }
}

// Antialias + L1 loss with the loss's gradient formed in the same pass, one
// thread per pixel, from a stored colour image: the form for the launches that
// batch_fit_kernel does not take (fit_words_bytes).  Every pixel: its output and
// |error| partial
// as batch_aa_l1_kernel computes them.  Then, for the pixels no blending pair
// touches (the listed ones belong to batch_aa_bwd_kernel, which forms
// the sign from the output and the target), the pixel's whole backward with
// the upstream gradient sign(out - target) * scale: interpolation backward
// (attribute gradients) and rasterisation backward (vertex gradients),
// reduced over runs of one triangle in the warp and scattered with float4
// atomics -- the work batch_bwd_kernel does for those pixels, done while
// the pixel's rast row and signs are at hand, with no gradient image written
// or read back.  The signs pass between the two phases as two bit masks, so
// an item may have at most 32 channels (more: DRP_DEVERR_CHANNELS, and the
// item gets no gradient here).  Warps never straddle items (256-pixel blocks).
__global__ void __launch_bounds__(256, 4) batch_aa_l1_grad_kernel(BatchArgs a) {
    __shared__ float warp_sum[8];
    pdl_wait();
    pdl_launch_dependents();
    const int2 blk = a.pix_blocks[blockIdx.x];
    const drp_batch_item& it = a.items[blk.x];
    const int pix = blk.y * 256 + threadIdx.x;
    const int W = it.width, H = it.height, C = it.channels;
    const bool in = pix < W * H;
    const float4* R = reinterpret_cast<const float4*>(a.rast) + it.pixel_offset;
    // the backward's rast row and vertex indices, loaded first so that their
    // latency overlaps the antialias work
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    int t = -1, i0 = 0, i1 = 0, i2 = 0;
    if (in) {
        r = R[pix];
        t = checked_tri(r.w, a.tri + 3 * (long long)it.tri_first, it.tri_count, it.num_vertices, i0, i1, i2);
    }
    float s = 0.0f;
    unsigned bits = 0u, nz = 0u, ps = 0u;
    {
        int src[4];
        float wt[4];
        const bool any = aa_fwd_terms_row(R, a.aa_rec + it.prim_offset * 2, it.tri_count, W, H, pix, in, src, wt,
                                          &bits);  // all lanes: pairs shared along the row
        if (in) {
            const long long row = it.image_offset + (long long)pix * C;
            s = aa_l1_channels(a.color + it.image_offset, C, pix, src, wt, any, a.target + row, a.l1_scale,
                               a.out + row, nullptr, &nz, &ps);
        }
    }
    aa_note_pixel<false>(a, it.pixel_offset + pix, in, bits);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = s;
    // the block's loss partial is added at the end: a barrier here would hold
    // every warp's backward until the slowest antialias pixel of the block
    pixel_backward_l1(a, it, pix, r, (bits == 0u && C <= 32) ? t : -1, i0, i1, i2, nz, ps);
    if (C > 32 && threadIdx.x == 0) atomicOr(a.stats + 2, DRP_DEVERR_CHANNELS);
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += warp_sum[w];
        a.block_loss[blockIdx.x] = t;
    }
}

// Interpolated colours of every pixel from its rast row: what the fine raster
// stores when it is asked to, for a backward that needs them after
// drp_batch_fit_l1 kept none.  Bound by its rast reads and colour writes.
__global__ void __launch_bounds__(256) batch_color_kernel(BatchArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    const int2 blk = a.pix_blocks[blockIdx.x];
    const drp_batch_item& it = a.items[blk.x];
    const int pix = blk.y * 256 + threadIdx.x, C = it.channels;
    if (pix >= it.width * it.height) return;
    const float4 r = reinterpret_cast<const float4*>(a.rast)[it.pixel_offset + pix];
    int i0 = 0, i1 = 0, i2 = 0;
    const int t = checked_tri(r.w, a.tri + 3 * (long long)it.tri_first, it.tri_count, it.num_vertices, i0, i1, i2);
    const float* A = a.attr + it.attr_offset;
    float* o = a.color + it.image_offset + (long long)pix * C;
    const bool vec = (C & 3) == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(o)) & 15) == 0;
    for (int c = 0; c < C; c += 4) {
        float x0[4], x1[4], x2[4], v[4];
        if (vec) {
            lerp_group<true>(A, C, c, t, i0, i1, i2, r.x, r.y, x0, x1, x2, v);
            store4<true>(o + c, C - c, v);
        } else {
            lerp_group<false>(A, C, c, t, i0, i1, i2, r.x, r.y, x0, x1, x2, v);
            store4<false>(o + c, C - c, v);
        }
    }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
struct BatchLayout {
    size_t stats, queue, prims, count, offset, cursor, chunks, list, aa, total;
};

BatchLayout batch_layout(long long total_prims, long long total_tiles, unsigned long long cap) {
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    BatchLayout L;
    L.stats = 0;
    L.queue = 64;
    L.prims = 256;
    L.count = up(L.prims + (size_t)total_prims * 48);
    L.offset = up(L.count + (size_t)total_tiles * 4);
    L.cursor = up(L.offset + (size_t)total_tiles * 4);
    L.chunks = up(L.cursor + (size_t)total_tiles * 4);
    // the antialias records sit before the list: their offset must not depend
    // on the list capacity (the backward may reuse the forward's records)
    L.aa = up(L.chunks + (size_t)scan_chunks(total_tiles) * 8);
    L.list = up(L.aa + (size_t)total_prims * 32);
    L.total = up(L.list + (size_t)cap * 4);
    return L;
}

// Antialias state block: list count at 0, per-pixel flags at 256, the pixel
// list (int32) after them.  No entry is told the block's size, so this layout
// belongs to the ABI version: scratch that a later form wants goes elsewhere.
static size_t aa_state_bytes(long long total_pixels, size_t* list_off) {
    const size_t flags_end = 256 + (size_t)total_pixels;
    const size_t lo = (flags_end + 255) / 256 * 256;
    if (list_off) *list_off = lo;
    return lo + (size_t)total_pixels * 4;
}

// Pixel words of batch_fit_kernel: they follow the workspace, whose size the
// entries are told; none where batch_aa_l1_grad_kernel's step is the faster.  A
// region is half a 32-pixel tile, but two 16-pixel or eight 8-pixel ones, whose other
// CTAs come and go for nothing; a walk pays by the pixels its columns stay in a
// triangle; more than eight channels go row by row (fit_rows), whose sums collide on
// few vertices (a plain multiple of eight has the fewest passes, four more than that a
// pass of their own).  Step over the other form's, smooth meshes of 24, 10, 3 and 1
// pixels a triangle and a coarse one (1280 triangles):
//   32-pixel tiles, 1.0M pixels:  1 channel 1.01 1.06 1.09 1.05 0.96, 4 0.95 1.01 1.03
//     1.03 0.92, 8 0.91 0.96 0.97 1.00 0.85, 9 0.86 0.92 0.88 0.92 1.13, 12 1.06 1.07
//     1.05 1.02 1.13, 20 1.00 1.01 0.96 0.97 1.02, 32 0.8
//   and 2.4M:  1 0.94 1.00 0.99 1.00 0.84, 4 0.9, 8 0.9, 9 0.8 (coarse 1.04), 12 1.0;
//     8.4M and 24 pixels a triangle: 0.7 to 0.9
//   16-pixel tiles, 1.0M:  1 1.10 1.15 1.17 1.17, 4 1.01 1.06 1.11 1.10, 8 1.02 1.07 1.09
//     1.07 0.91, 12 1.2, 16 1.1;  1.7M:  1 1.03 1.06 1.11 1.10 0.84, 4 0.97 1.00 1.03
//     1.05 0.86, 8 0.93 0.98 1.00 1.03 0.82, 13 0.8 (coarse 1.2), 12 1.1, 16 1.04;
//     4.2M:  4 0.93 0.96 0.98 0.99, 12 1.05, 16 0.95
//   8-pixel tiles, 4.2M:  1 1.1, 4 1.01 1.06 1.03 1.03, 8 0.98 1.04 1.02, 13 0.83, 12 1.1
// (Rough meshes, a silhouette at most pixels, up to 0.1 more.)
static size_t fit_words_bytes(long long pixels, long long image_floats, long long prims, int tile_log2) {
    constexpr long long kMi = 1ll << 20, kNever = 1ll << 62;
    if (pixels < kFitPixels) return 0;
    const long long C = (image_floats + pixels - 1) / pixels;
    long long from = kNever, per_prim = 0;  // pixels of the launch, pixels per triangle
    bool coarse = true;                     // also with more than 256 pixels per triangle
    if (C <= 8) {
        if (tile_log2 == 5) {
            from = kMi;
            if (C <= 2) per_prim = 2 * pixels < 3 * kMi ? 32 : (pixels < 2 * kMi ? 16 : 0);
            else if (C <= 5) per_prim = 4 * pixels < 5 * kMi ? 12 : 0;
        } else if (tile_log2 == 4) {
            const bool few = 4 * pixels < 5 * kMi;
            from = !few || C == 3 || C >= 5 ? kMi : kNever;
            per_prim = few ? (C == 3 ? 64 : 32) : (C <= 2 ? 48 : (C <= 5 ? 16 : 4));
        } else if (C >= 3) {
            from = 4 * kMi;
            per_prim = C <= 5 ? 48 : 16;
        }
    } else if (C % 8 == 0) {
        if (tile_log2 == 5 || C >= 32) from = kMi;
        else if (tile_log2 == 4) from = C >= 24 ? 3 * kMi / 2 : 2 * kMi;
    } else {
        coarse = false;
        if (tile_log2 == 5) from = C == 12 ? 2 * kMi : (C % 4 == 0 ? 5 * kMi / 4 : kMi);
        else if (C % 4 != 0) from = tile_log2 == 4 ? 5 * kMi / 4 : 4 * kMi;
        else if (tile_log2 == 4 && C > 12) from = 2 * kMi;
    }
    const bool fit = pixels >= from && per_prim * prims <= pixels && (coarse || 256 * prims >= pixels);
    return fit ? (size_t)pixels * 4 : 0;
}

static void carve_aa_state(BatchArgs& a, void* state, long long total_pixels) {
    if (!state) return;
    size_t lo = 0;
    aa_state_bytes(total_pixels, &lo);
    char* p = static_cast<char*>(state);
    a.aa_count = reinterpret_cast<unsigned*>(p);
    a.aa_flags = reinterpret_cast<unsigned char*>(p + 256);
    a.aa_list = reinterpret_cast<int*>(p + lo);
}

static void carve(BatchArgs& a, void* ws, const BatchLayout& L) {
    char* w = static_cast<char*>(ws);
    a.stats = reinterpret_cast<uint32_t*>(w + L.stats);
    a.queue = reinterpret_cast<uint32_t*>(w + L.queue);
    a.loss_count = a.stats + 32;  // in the stats block, zeroed with it
    a.prims = reinterpret_cast<int4*>(w + L.prims);
    a.tile_count = reinterpret_cast<uint32_t*>(w + L.count);
    a.tile_offset = reinterpret_cast<uint32_t*>(w + L.offset);
    a.tile_cursor = reinterpret_cast<uint32_t*>(w + L.cursor);
    a.tile_list = reinterpret_cast<uint32_t*>(w + L.list);
    a.chunk_sums = reinterpret_cast<unsigned long long*>(w + L.chunks);
    a.aa_rec = reinterpret_cast<float4*>(w + L.aa);
}

// Rows per warp: a walk of eight adds fewest sums per pixel, but below this
// many regions two warps each leave the chip idle, and four rows per warp are
// faster (one 1024 x 1024 view, 2048 regions: 126.7 against 129.5 us per step;
// 64 views of 512 x 512, 32768 regions: 1039 against 946 us).
constexpr long long kFitTallRegions = 4096;

// Rows per warp of batch_blend_kernel: four read fewer words twice, but below
// this many pixels two finish sooner -- the longest chain is that of the warp
// with the most blends (344,438 pixels of small dense meshes: 217 with two,
// 224 with four, 238 us with eight; 565,312: 157, 163, 174; 1,991,582: 422,
// 420, 430; 5,848,746: 618, 591, 608).
constexpr long long kBlendTallPixels = 1ll << 20;

// Up to this many tiles per resident fine CTA the work order is sorted.
constexpr long long kOrderTilesPerCTA = 8;

// Zeroes the stats / work-queue block (256 bytes), the antialias pixel-list
// count and the per-tile counts that a forward accumulates into: one kernel
// in the forward's launch chain instead of three memsets.
// Also zeroes `zero_n` floats at `zero` (the gradient buffers of
// drp_batch_forward_l1_grad, when the call is asked to start them at zero).
__global__ void __launch_bounds__(256) batch_clear_kernel(uint32_t* stats, unsigned* aa_count,
                                                          uint32_t* tile_count, long long tiles, float* zero,
                                                          long long zero_n) {
    pdl_wait();
    pdl_launch_dependents();
    const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    if (i0 < 64) stats[i0] = 0u;
    if (i0 == 0 && aa_count) *aa_count = 0u;
    for (long long i = i0; i < tiles; i += stride) tile_count[i] = 0u;
    if (zero) {
        // 16-byte groups from the first aligned float (the buffer start is
        // at least 4-byte aligned), scalar head and tail
        const long long head = (long long)(((16 - (reinterpret_cast<uintptr_t>(zero) & 15)) & 15) >> 2);
        const long long h = head < zero_n ? head : zero_n;
        if (i0 < h) zero[i0] = 0.f;
        float4* z4 = reinterpret_cast<float4*>(zero + h);
        const long long n4 = (zero_n - h) >> 2;
        for (long long i = i0; i < n4; i += stride) z4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const long long t0 = h + 4 * n4;
        if (i0 < zero_n - t0) zero[t0 + i0] = 0.f;
    }
}

template <int TL, int TPT, bool FIT, int NT = fine_threads<TL>()>
static void launch_batch_fine(const BatchArgs& a, cudaStream_t s) {
    // persistent grid: every resident CTA slot of the device (occupancy per
    // kernel instantiation is device-independent for one architecture)
    static std::atomic<int> per_sm{0};
    int per = per_sm.load(std::memory_order_relaxed);
    if (per == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, batch_fine_kernel<TL, TPT, FIT, NT>, NT, 0);
        per = per > 0 ? per : 1;
        per_sm.store(per, std::memory_order_relaxed);
    }
    const int sms = drp_current_sm_count();
    const long long grid = (long long)(sms > 0 ? sms : 1) * per;
    const long long g = a.total_tiles < grid ? a.total_tiles : grid;
    if (g <= 0) return;
    // With a few tiles per resident CTA, hand the longest tile lists out
    // first (the order goes into the fill cursors, which are spent by now).
    BatchArgs b = a;
    b.tile_order = nullptr;
    if (a.total_tiles > g && a.total_tiles <= kOrderTilesPerCTA * grid) {
        launch_tile_order(a.tile_count, a.total_tiles, a.tile_cursor, s);
        b.tile_order = a.tile_cursor;
    }
    launch_pdl(batch_fine_kernel<TL, TPT, FIT, NT>, dim3((unsigned)g), dim3(NT), s, b);
    drp_note_launch();
}

template <int TL, bool FIT>
static void launch_batch_fine(const BatchArgs& a, cudaStream_t s) {
    switch (a.tpt) {
    case 0:
        if (fine_many(TL, a.total_tiles, a.total_prims)) launch_batch_fine<TL, 0, FIT, fine_threads_many<TL>()>(a, s);
        else launch_batch_fine<TL, 0, FIT>(a, s);
        break;
    case 1: launch_batch_fine<TL, 1, FIT>(a, s); break;
    case 2: launch_batch_fine<TL, 2, FIT>(a, s); break;
    case 4: launch_batch_fine<TL, 4, FIT>(a, s); break;
    case 8: launch_batch_fine<TL, 8, FIT>(a, s); break;
    case 16: launch_batch_fine<TL, 16, FIT>(a, s); break;
    default: launch_batch_fine<TL, 32, FIT>(a, s); break;
    }
}

template <int TL>
static void launch_batch_raster(const BatchArgs& a, cudaStream_t s) {
    constexpr int kSplit = setup_split(kSetupCount), kTris = 256 / kSplit, kFillSplit = setup_split(kSetupFill);
    if (a.n_prim_blocks > 0 && a.bin_depth) {
        launch_pdl(batch_setup_bin_kernel<TL, kSetupBins>, dim3((unsigned)(a.n_prim_blocks * kSplit)),
                   dim3(a.aa_records ? 2 * kTris : kTris), s, a);
        drp_note_launch();
    } else if (a.n_prim_blocks > 0) {
        launch_pdl(batch_setup_bin_kernel<TL, kSetupCount>, dim3((unsigned)(a.n_prim_blocks * kSplit)),
                   dim3(a.aa_records ? 2 * kTris : kTris), s, a);
        drp_note_launch();
        launch_tile_scan(a.tile_count, a.tile_offset, a.tile_cursor, a.total_tiles, a.chunk_sums,
                         reinterpret_cast<unsigned long long*>(a.stats), s);
        batch_setup_bin_kernel<TL, kSetupFill><<<(unsigned)(a.n_prim_blocks * kFillSplit), 256 / kFillSplit, 0, s>>>(a);
        drp_note_launch();
    } else {
        cudaMemsetAsync(a.tile_offset, 0, sizeof(uint32_t) * a.total_tiles, s);
    }
    if (a.fit) launch_batch_fine<TL, true>(a, s);
    else launch_batch_fine<TL, false>(a, s);
}

// A side stream with its fork / join events, one per host thread and device,
// created on first use outside stream capture (inside a capture, before the
// first ordinary call, the caller's stream serves alone).  Captured forks
// and joins become graph edges.  The caller's stream belongs to the current
// device, as for every launch of this library (a stream query here would
// invalidate a capture in progress).
struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};

static bool side_stream(cudaStream_t s, SideStream& out) {
    constexpr int kMaxDev = 64;
    thread_local SideStream cache[kMaxDev];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) {
        cudaGetLastError();
        return false;
    }
    SideStream& c = cache[dev];
    if (!c.stream) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
            cudaGetLastError();
            return false;
        }
        SideStream n;
        if (cudaStreamCreateWithFlags(&n.stream, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&n.fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&n.join, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            if (n.stream) cudaStreamDestroy(n.stream);
            if (n.fork) cudaEventDestroy(n.fork);
            return false;
        }
        c = n;
    }
    out = c;
    return true;
}

template <int ROWS>
static void launch_blend(const BatchArgs& a, long long regions, cudaStream_t s) {
    const long long units = 16 / ROWS * regions;
    launch_pdl(batch_blend_kernel<ROWS>, dim3((unsigned)((units + kBlendWarps - 1) / kBlendWarps)),
               dim3(32 * kBlendWarps), s, a);
    drp_note_launch();
}

int launch_batch_forward(BatchArgs a, void* ws, const BatchLayout& L, cudaStream_t s) {
    carve(a, ws, L);
    {
        // stats and work queue, list count, tile counts (and the buffers a
        // gradient-forming forward is asked to zero)
        long long need = a.total_tiles > 64 ? a.total_tiles : 64;
        if (a.zero_first && a.zero_floats / 4 > need) need = a.zero_floats / 4;
        const int sms = drp_current_sm_count();
        long long blocks = (need + 255) / 256;
        const long long cap = (long long)(sms > 0 ? sms : 1) * 4;
        if (blocks > cap) blocks = cap;
        launch_pdl(batch_clear_kernel, dim3((unsigned)blocks), dim3(256), s, a.stats, a.aa_count, a.tile_count,
                   (long long)a.total_tiles, a.zero_first, a.zero_floats);
        drp_note_launch();
    }
    switch (a.tile_log2) {
    case 3: launch_batch_raster<3>(a, s); break;
    case 5: launch_batch_raster<5>(a, s); break;
    default: launch_batch_raster<4>(a, s); break;
    }
    // (the antialias triangle records were written by the setup / count pass)
    if (a.target && a.l1_grads) {
        if (a.n_pix_blocks > 0) {
            if (a.fit) {
                const long long regions = a.total_tiles * fit_regions_per_tile(a.tile_log2);
                if (regions < kFitTallRegions)
                    launch_pdl(batch_fit_kernel<4>, dim3((unsigned)regions), dim3(128), s, a);
                else
                    launch_pdl(batch_fit_kernel<2>, dim3((unsigned)regions), dim3(64), s, a);
            } else {
                launch_pdl(batch_aa_l1_grad_kernel, dim3((unsigned)a.n_pix_blocks), dim3(256), s, a);
            }
            drp_note_launch();
            // the listed pixels' whole backward, and the final loss sum
            // (the last block's, or fit_loss by all): one launch on the chain
            if (a.fit)
                launch_pdl(batch_aa_bwd_kernel<kListFit, kListLanes>,
                           dim3((unsigned)list_kernel_grid<kListFit>(a.n_pix_blocks)), dim3(256), s, a);
            else
                launch_pdl(batch_aa_bwd_kernel<kListL1, kListLanes>,
                           dim3((unsigned)list_kernel_grid<kListL1>(a.n_pix_blocks)), dim3(256), s, a);
            drp_note_launch();
        } else {
            launch_l1_final(a.block_loss, a.n_pix_blocks, a.l1_scale, a.loss, s);
        }
        return 0;
    }
    if (a.target) {
        if (a.n_pix_blocks > 0) {
            launch_pdl(batch_aa_l1_kernel, dim3((unsigned)a.n_pix_blocks), dim3(256), s, a);
            drp_note_launch();
        }
        launch_l1_final(a.block_loss, a.n_pix_blocks, a.l1_scale, a.loss, s);
        return 0;
    }
    if (a.fit) {
        if (a.n_pix_blocks > 0) {
            const long long regions = a.total_tiles * fit_regions_per_tile(a.tile_log2);
            if (a.total_pixels < kBlendTallPixels) launch_blend<2>(a, regions, s);
            else launch_blend<4>(a, regions, s);
        }
        return 0;
    }
    if (!a.out) return 0;  // raster + interpolation only (recomputing them for the backward)
    if (a.n_pix_blocks > 0) {
        launch_pdl(batch_aa_fwd_kernel, dim3((unsigned)a.n_pix_blocks), dim3(256), s, a);
        drp_note_launch();
    }
    return 0;
}

int launch_batch_backward(BatchArgs a, void* ws, const BatchLayout& L, bool reuse_records, cudaStream_t s) {
    carve(a, ws, L);
    if (a.n_prim_blocks > 0 && !reuse_records) {
        launch_pdl(batch_aa_setup_kernel, dim3((unsigned)a.n_prim_blocks), dim3(256), s, a);
        drp_note_launch();
    }
    if (a.n_pix_blocks <= 0) return 0;
    if (!a.aa_flags) {
        batch_bwd_kernel<<<(unsigned)a.n_pix_blocks, 256, 0, s>>>(a);
        drp_note_launch();
        return 0;
    }
    // The listed pixels' kernel (latency-bound, a few percent of the pixels)
    // and the fused backward of all other pixels are independent: fork the
    // list kernel onto a side stream so it fills the SMs beside the main
    // kernel and its tail, then join.  Both only add into the gradients.
    const long long g = list_kernel_grid<kListBackward>(a.n_pix_blocks);
    SideStream side;
    const bool fork = side_stream(s, side);
    if (fork) {
        cudaEventRecord(side.fork, s);
        cudaStreamWaitEvent(side.stream, side.fork, 0);
    }
    batch_bwd_kernel<<<(unsigned)a.n_pix_blocks, 256, 0, s>>>(a);
    drp_note_launch();
    batch_aa_bwd_kernel<kListBackward, kListLanes><<<(unsigned)g, 256, 0, fork ? side.stream : s>>>(a);
    drp_note_launch();
    if (fork) {
        cudaEventRecord(side.join, side.stream);
        cudaStreamWaitEvent(s, side.join, 0);
    }
    return 0;
}

}  // namespace drp

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
#define DRP_API extern "C" __attribute__((visibility("default")))

namespace {
int bfail(const char* msg) {
    drp_set_last_error(msg);
    return DRP_STATUS_INVALID_ARGUMENT;
}
}  // namespace

DRP_API int drp_batch_plan(drp_batch_item* items, int num_items, int tile_log2, long long* totals) {
    if (!items || num_items <= 0 || !totals) return bfail("drp_batch_plan: bad arguments");
    if (tile_log2 < 3 || tile_log2 > 5) return bfail("drp_batch_plan: tile_log2 must be 3, 4 or 5");
    long long prims = 0, tiles = 0, pixels = 0, floats = 0, pblocks = 0, xblocks = 0;
    for (int i = 0; i < num_items; ++i) {
        drp_batch_item& it = items[i];
        if (it.height <= 0 || it.width <= 0 || it.height > DRP_MAX_RESOLUTION || it.width > DRP_MAX_RESOLUTION ||
            it.channels <= 0 || it.tri_count < 0 || it.tri_first < 0 || it.num_vertices < 0 || it.pos_offset < 0 ||
            it.attr_offset < 0)
            return bfail("drp_batch_plan: item with invalid size, resolution or offset");
        it.tiles_x = (it.width + (1 << tile_log2) - 1) >> tile_log2;
        it.tiles_y = (it.height + (1 << tile_log2) - 1) >> tile_log2;
        it.prim_offset = prims;
        it.tile_offset = tiles;
        it.pixel_offset = pixels;
        it.image_offset = floats;
        prims += it.tri_count;
        tiles += (long long)it.tiles_x * it.tiles_y;
        pixels += (long long)it.width * it.height;
        floats += (long long)it.width * it.height * it.channels;
        pblocks += (it.tri_count + 255) / 256;
        xblocks += ((long long)it.width * it.height + 255) / 256;
    }
    totals[0] = prims;
    totals[1] = tiles;
    totals[2] = pixels;
    totals[3] = floats;
    totals[4] = pblocks;
    totals[5] = xblocks;
    return DRP_STATUS_OK;
}

DRP_API int drp_batch_block_maps(const drp_batch_item* items, int num_items, int* prim_block_map,
                                 int* pixel_block_map) {
    if (!items || num_items <= 0 || !prim_block_map || !pixel_block_map) return bfail("drp_batch_block_maps: null");
    long long p = 0, x = 0;
    for (int i = 0; i < num_items; ++i) {
        const long long nb = (items[i].tri_count + 255) / 256;
        for (long long k = 0; k < nb; ++k, ++p) {
            prim_block_map[2 * p] = i;
            prim_block_map[2 * p + 1] = (int)k;
        }
        const long long xb = ((long long)items[i].width * items[i].height + 255) / 256;
        for (long long k = 0; k < xb; ++k, ++x) {
            pixel_block_map[2 * x] = i;
            pixel_block_map[2 * x + 1] = (int)k;
        }
    }
    return DRP_STATUS_OK;
}

DRP_API int drp_batch_aa_state_size(long long total_pixels, size_t* bytes) {
    if (!bytes || total_pixels <= 0) return bfail("drp_batch_aa_state_size: bad arguments");
    *bytes = drp::aa_state_bytes(total_pixels, nullptr);
    return DRP_STATUS_OK;
}

DRP_API int drp_batch_fit_words_size(long long total_pixels, long long image_floats, long long total_prims,
                                     int tile_log2, size_t* bytes) {
    if (!bytes || total_pixels <= 0 || image_floats < total_pixels || total_prims < 0 || tile_log2 < 3 ||
        tile_log2 > 5)
        return bfail("drp_batch_fit_words_size: bad arguments");
    *bytes = drp::fit_words_bytes(total_pixels, image_floats, total_prims, tile_log2);
    return DRP_STATUS_OK;
}

DRP_API int drp_batch_workspace_size(long long total_prims, long long total_tiles, unsigned long long list_capacity,
                                     size_t* bytes) {
    if (!bytes || total_prims < 0 || total_tiles < 0 || list_capacity > 0x7fffffffull)
        return bfail("drp_batch_workspace_size: bad arguments");
    *bytes = drp::batch_layout(total_prims, total_tiles, list_capacity).total;
    return DRP_STATUS_OK;
}

static int batch_common(void* ws, size_t ws_bytes, const drp_batch_item* items, int num_items,
                        const int* prim_block_map, long long prim_blocks, const int* pixel_block_map,
                        long long pixel_blocks, long long total_prims, long long total_tiles,
                        unsigned long long list_capacity, const float* pos, const int* tri, const float* attr,
                        drp::BatchArgs& a, drp::BatchLayout& L) {
    if (!ws || (reinterpret_cast<uintptr_t>(ws) & 255)) return bfail("batch: workspace must be 256-byte aligned");
    if (!items || num_items <= 0 || !pos || !tri || !attr) return bfail("batch: null table or buffer");
    if ((prim_blocks > 0 && !prim_block_map) || (pixel_blocks > 0 && !pixel_block_map) || prim_blocks < 0 ||
        pixel_blocks < 0 || prim_blocks > 0x7fffffffll / drp::kSetupSplitMost || pixel_blocks > 0x7fffffffll)
        return bfail("batch: bad block maps");
    if ((reinterpret_cast<uintptr_t>(pos) & 15)) return bfail("batch: pos must be 16-byte aligned");
    if (list_capacity > 0x7fffffffull) return bfail("batch: list_capacity above 2^31 - 1");
    L = drp::batch_layout(total_prims, total_tiles, list_capacity);
    if (ws_bytes < L.total) {
        drp_set_last_error("batch: workspace too small");
        return DRP_STATUS_WORKSPACE_TOO_SMALL;
    }
    a = drp::BatchArgs{};
    a.items = items;
    a.num_items = num_items;
    a.prim_blocks = reinterpret_cast<const int2*>(prim_block_map);
    a.n_prim_blocks = prim_blocks;
    a.pix_blocks = reinterpret_cast<const int2*>(pixel_block_map);
    a.n_pix_blocks = pixel_blocks;
    a.total_prims = total_prims;
    a.total_tiles = total_tiles;
    a.pos = pos;
    a.tri = tri;
    a.attr = attr;
    a.list_capacity = list_capacity;
    return DRP_STATUS_OK;
}

DRP_API int drp_batch_forward(void* workspace, size_t workspace_bytes, const drp_batch_item* items, int num_items,
                              const int* prim_block_map, long long prim_blocks, const int* pixel_block_map,
                              long long pixel_blocks, long long total_prims, long long total_tiles, const float* pos,
                              const int* tri, const float* attr, const int* nbr, int tile_log2, int threads_per_tri,
                              unsigned long long list_capacity, unsigned bin_depth, float* rast, float* color,
                              float* out, void* aa_state, long long total_pixels, void* stream) {
    drp::BatchArgs a;
    drp::BatchLayout L;
    int st = batch_common(workspace, workspace_bytes, items, num_items, prim_block_map, prim_blocks, pixel_block_map,
                          pixel_blocks, total_prims, total_tiles, list_capacity, pos, tri, attr, a, L);
    if (st) return st;
    if (tile_log2 < 3 || tile_log2 > 5) return bfail("batch: tile_log2 must be 3, 4 or 5");
    if (threads_per_tri < 0 || threads_per_tri > 32 || (threads_per_tri & (threads_per_tri - 1)))
        return bfail("batch: threads_per_tri must be 0 or a power of two <= 32");
    if (!rast || !color || (reinterpret_cast<uintptr_t>(rast) & 15)) return bfail("batch: bad outputs");
    if (bin_depth && (unsigned long long)total_tiles * bin_depth > list_capacity)
        return bfail("batch: list_capacity below total_tiles * bin_depth");
    a.nbr = nbr;
    a.tile_log2 = tile_log2;
    a.tpt = threads_per_tri;
    a.bin_depth = bin_depth;
    a.rast = rast;
    a.color = color;
    a.out = out;
    if (aa_state && ((reinterpret_cast<uintptr_t>(aa_state) & 255) || total_pixels <= 0))
        return bfail("batch: aa_state must be 256-byte aligned, with total_pixels > 0");
    carve_aa_state(a, aa_state, total_pixels);
    a.emit_out = out != nullptr;
    a.aa_records = out != nullptr;  // raster only: no antialias pass, no records
    drp::launch_batch_forward(a, workspace, L, static_cast<cudaStream_t>(stream));
    return drp_check_launch("drp_batch_forward");
}

DRP_API int drp_batch_render(void* workspace, size_t workspace_bytes, const drp_batch_item* items, int num_items,
                             const int* prim_block_map, long long prim_blocks, const int* pixel_block_map,
                             long long pixel_blocks, long long total_prims, long long total_tiles, const float* pos,
                             const int* tri, const float* attr, const int* nbr, int tile_log2, int threads_per_tri,
                             unsigned long long list_capacity, unsigned bin_depth, float* rast, void* words,
                             float* out, long long total_pixels, void* stream) {
    drp::BatchArgs a;
    drp::BatchLayout L;
    int st = batch_common(workspace, workspace_bytes, items, num_items, prim_block_map, prim_blocks, pixel_block_map,
                          pixel_blocks, total_prims, total_tiles, list_capacity, pos, tri, attr, a, L);
    if (st) return st;
    if (tile_log2 < 3 || tile_log2 > 5) return bfail("batch: tile_log2 must be 3, 4 or 5");
    if (threads_per_tri < 0 || threads_per_tri > 32 || (threads_per_tri & (threads_per_tri - 1)))
        return bfail("batch: threads_per_tri must be 0 or a power of two <= 32");
    if (!rast || !words || !out || total_pixels <= 0 || (reinterpret_cast<uintptr_t>(rast) & 15) ||
        (reinterpret_cast<uintptr_t>(words) & 3))
        return bfail("batch: bad outputs");
    if (bin_depth && (unsigned long long)total_tiles * bin_depth > list_capacity)
        return bfail("batch: list_capacity below total_tiles * bin_depth");
    a.nbr = nbr;
    a.tile_log2 = tile_log2;
    a.tpt = threads_per_tri;
    a.bin_depth = bin_depth;
    a.rast = rast;
    a.color = out;  // the fine raster writes the colours in place
    a.out = out;
    a.aa_words = static_cast<uint32_t*>(words);
    a.total_pixels = total_pixels;
    a.fit = true;
    a.emit_color = true;
    a.emit_out = false;
    a.aa_records = true;
    drp::launch_batch_forward(a, workspace, L, static_cast<cudaStream_t>(stream));
    return drp_check_launch("drp_batch_render");
}

DRP_API int drp_batch_forward_l1(void* workspace, size_t workspace_bytes, const drp_batch_item* items, int num_items,
                                 const int* prim_block_map, long long prim_blocks, const int* pixel_block_map,
                                 long long pixel_blocks, long long total_prims, long long total_tiles,
                                 const float* pos, const int* tri, const float* attr, const int* nbr, int tile_log2,
                                 int threads_per_tri, unsigned long long list_capacity, unsigned bin_depth,
                                 float* rast, float* color, float* out, void* aa_state, long long total_pixels,
                                 const float* target, float scale, float* grad, float* block_loss, float* loss,
                                 void* stream) {
    drp::BatchArgs a;
    drp::BatchLayout L;
    int st = batch_common(workspace, workspace_bytes, items, num_items, prim_block_map, prim_blocks, pixel_block_map,
                          pixel_blocks, total_prims, total_tiles, list_capacity, pos, tri, attr, a, L);
    if (st) return st;
    if (tile_log2 < 3 || tile_log2 > 5) return bfail("batch: tile_log2 must be 3, 4 or 5");
    if (threads_per_tri < 0 || threads_per_tri > 32 || (threads_per_tri & (threads_per_tri - 1)))
        return bfail("batch: threads_per_tri must be 0 or a power of two <= 32");
    if (!rast || !color || !target || !grad || !loss || (pixel_blocks > 0 && !block_loss) ||
        (reinterpret_cast<uintptr_t>(rast) & 15))
        return bfail("batch: bad outputs");
    if (bin_depth && (unsigned long long)total_tiles * bin_depth > list_capacity)
        return bfail("batch: list_capacity below total_tiles * bin_depth");
    a.nbr = nbr;
    a.tile_log2 = tile_log2;
    a.tpt = threads_per_tri;
    a.bin_depth = bin_depth;
    a.rast = rast;
    a.color = color;
    a.out = out;
    if (aa_state && ((reinterpret_cast<uintptr_t>(aa_state) & 255) || total_pixels <= 0))
        return bfail("batch: aa_state must be 256-byte aligned, with total_pixels > 0");
    carve_aa_state(a, aa_state, total_pixels);
    a.emit_out = false;  // the fused antialias + loss pass writes every output pixel
    a.aa_records = true;
    a.target = target;
    a.l1_scale = scale;
    a.l1_grad = grad;
    a.block_loss = block_loss;
    a.loss = loss;
    drp::launch_batch_forward(a, workspace, L, static_cast<cudaStream_t>(stream));
    return drp_check_launch("drp_batch_forward_l1");
}

static int batch_fit_l1(const char* who, bool full_color, void* workspace, size_t workspace_bytes,
                        const drp_batch_item* items, int num_items, const int* prim_block_map, long long prim_blocks,
                        const int* pixel_block_map, long long pixel_blocks, long long total_prims,
                        long long total_tiles, const float* pos, const int* tri, const float* attr,
                        const int* nbr, int tile_log2, int threads_per_tri,
                        unsigned long long list_capacity, unsigned bin_depth, float* rast, float* color,
                        float* out, void* aa_state, long long total_pixels, const float* target,
                        float scale, float* block_loss, float* loss, float* grad_pos, float* grad_attr,
                        float* zero_first, long long zero_floats, void* stream) {
    drp::BatchArgs a;
    drp::BatchLayout L;
    int st = batch_common(workspace, workspace_bytes, items, num_items, prim_block_map, prim_blocks, pixel_block_map,
                          pixel_blocks, total_prims, total_tiles, list_capacity, pos, tri, attr, a, L);
    if (st) return st;
    if (tile_log2 < 3 || tile_log2 > 5) return bfail("batch: tile_log2 must be 3, 4 or 5");
    if (threads_per_tri < 0 || threads_per_tri > 32 || (threads_per_tri & (threads_per_tri - 1)))
        return bfail("batch: threads_per_tri must be 0 or a power of two <= 32");
    if (!rast || !color || !out || !target || !loss || (pixel_blocks > 0 && !block_loss) ||
        (reinterpret_cast<uintptr_t>(rast) & 15))
        return bfail("batch: bad outputs");
    if (!grad_pos || !grad_attr || (reinterpret_cast<uintptr_t>(grad_pos) & 15))
        return bfail("batch: bad gradient buffers");
    if (!aa_state || (reinterpret_cast<uintptr_t>(aa_state) & 255) || total_pixels <= 0)
        return bfail("batch: the gradient pass needs the antialias state (256-byte aligned, total_pixels > 0)");
    if (bin_depth && (unsigned long long)total_tiles * bin_depth > list_capacity)
        return bfail("batch: list_capacity below total_tiles * bin_depth");
    a.nbr = nbr;
    a.tile_log2 = tile_log2;
    a.tpt = threads_per_tri;
    a.bin_depth = bin_depth;
    a.rast = rast;
    a.color = color;
    a.out = out;
    carve_aa_state(a, aa_state, total_pixels);
    // room for the pixel words chooses the form (fit_words_bytes)
    a.fit = total_pixels >= drp::kFitPixels && workspace_bytes >= L.total + (size_t)total_pixels * 4;
    a.aa_words = a.fit ? reinterpret_cast<uint32_t*>(static_cast<char*>(workspace) + L.total) : nullptr;
    a.emit_color = full_color;  // else the loss pass stores the listed pixels' colours only
    a.emit_out = false;  // the fused antialias + loss pass writes every output pixel
    a.aa_records = true;
    a.target = target;
    a.l1_scale = scale;
    a.l1_grad = nullptr;
    a.block_loss = block_loss;
    a.loss = loss;
    a.l1_grads = true;
    a.grad_pos = grad_pos;
    a.grad_attr = grad_attr;
    if (zero_floats < 0 || (zero_floats > 0 && !zero_first) || (reinterpret_cast<uintptr_t>(zero_first) & 3))
        return bfail("batch: bad zero region");
    a.zero_first = zero_floats > 0 ? zero_first : nullptr;
    a.zero_floats = zero_floats;
    drp::launch_batch_forward(a, workspace, L, static_cast<cudaStream_t>(stream));
    return drp_check_launch(who);
}

DRP_API int drp_batch_forward_l1_grad(void* workspace, size_t workspace_bytes, const drp_batch_item* items,
                                      int num_items, const int* prim_block_map, long long prim_blocks,
                                      const int* pixel_block_map, long long pixel_blocks, long long total_prims,
                                      long long total_tiles, const float* pos, const int* tri, const float* attr,
                                      const int* nbr, int tile_log2, int threads_per_tri,
                                      unsigned long long list_capacity, unsigned bin_depth, float* rast, float* color,
                                      float* out, void* aa_state, long long total_pixels, const float* target,
                                      float scale, float* block_loss, float* loss, float* grad_pos, float* grad_attr,
                                      float* zero_first, long long zero_floats, void* stream) {
    return batch_fit_l1("drp_batch_forward_l1_grad", true, workspace, workspace_bytes, items, num_items,
                        prim_block_map, prim_blocks, pixel_block_map, pixel_blocks, total_prims, total_tiles, pos, tri,
                        attr, nbr, tile_log2, threads_per_tri, list_capacity, bin_depth, rast, color, out, aa_state,
                        total_pixels, target, scale, block_loss, loss, grad_pos, grad_attr, zero_first, zero_floats,
                        stream);
}

DRP_API int drp_batch_fit_l1(void* workspace, size_t workspace_bytes, const drp_batch_item* items,
                             int num_items, const int* prim_block_map, long long prim_blocks,
                             const int* pixel_block_map, long long pixel_blocks, long long total_prims,
                             long long total_tiles, const float* pos, const int* tri, const float* attr,
                             const int* nbr, int tile_log2, int threads_per_tri,
                             unsigned long long list_capacity, unsigned bin_depth, float* rast, float* color,
                             float* out, void* aa_state, long long total_pixels, const float* target,
                             float scale, float* block_loss, float* loss, float* grad_pos, float* grad_attr,
                             float* zero_first, long long zero_floats, void* stream) {
    return batch_fit_l1("drp_batch_fit_l1", false, workspace, workspace_bytes, items, num_items, prim_block_map,
                        prim_blocks, pixel_block_map, pixel_blocks, total_prims, total_tiles, pos, tri, attr, nbr,
                        tile_log2, threads_per_tri, list_capacity, bin_depth, rast, color, out, aa_state,
                        total_pixels, target, scale, block_loss, loss, grad_pos, grad_attr, zero_first, zero_floats,
                        stream);
}

DRP_API int drp_batch_colors(const drp_batch_item* items, int num_items, const int* pixel_block_map,
                             long long pixel_blocks, const int* tri, const float* attr, const float* rast,
                             float* color, void* stream) {
    if (!items || num_items <= 0 || !tri || !attr || !rast || !color || (reinterpret_cast<uintptr_t>(rast) & 15) ||
        pixel_blocks < 0 || pixel_blocks > 0x7fffffffll || (pixel_blocks > 0 && !pixel_block_map))
        return bfail("drp_batch_colors: bad table or buffers");
    if (pixel_blocks == 0) return DRP_STATUS_OK;
    drp::BatchArgs a{};
    a.items = items;
    a.num_items = num_items;
    a.pix_blocks = reinterpret_cast<const int2*>(pixel_block_map);
    a.tri = tri;
    a.attr = attr;
    a.rast = const_cast<float*>(rast);
    a.color = color;
    drp::launch_pdl(drp::batch_color_kernel, dim3((unsigned)pixel_blocks), dim3(256),
                    static_cast<cudaStream_t>(stream), a);
    drp_note_launch();
    return drp_check_launch("drp_batch_colors");
}

DRP_API int drp_batch_backward(void* workspace, size_t workspace_bytes, const drp_batch_item* items, int num_items,
                               const int* prim_block_map, long long prim_blocks, const int* pixel_block_map,
                               long long pixel_blocks, long long total_prims, long long total_tiles,
                               const float* pos, const int* tri, const float* attr, const int* nbr,
                               const float* rast, const float* color, const void* aa_state, long long total_pixels,
                               float* aa_grad,
                               const float* grad_out, float* grad_pos, float* grad_attr, const float* grad_scale,
                               int flags, void* stream) {
    drp::BatchArgs a;
    drp::BatchLayout L;
    int st = batch_common(workspace, workspace_bytes, items, num_items, prim_block_map, prim_blocks, pixel_block_map,
                          pixel_blocks, total_prims, total_tiles, 0, pos, tri, attr, a, L);
    if (st) return st;
    if (!rast || !color || !grad_out || !grad_pos || !grad_attr || (reinterpret_cast<uintptr_t>(grad_pos) & 15))
        return bfail("batch: bad gradient buffers");
    a.nbr = nbr;
    a.rast = const_cast<float*>(rast);
    a.color = const_cast<float*>(color);
    (void)aa_grad;  // no longer used: the listed pixels' backward is fused into their kernel
    if (aa_state && ((reinterpret_cast<uintptr_t>(aa_state) & 255) || total_pixels <= 0))
        return bfail("batch: aa_state needs 256-byte alignment and total_pixels > 0");
    carve_aa_state(a, const_cast<void*>(aa_state), total_pixels);
    a.grad_out = grad_out;
    a.grad_pos = grad_pos;
    a.grad_attr = grad_attr;
    a.grad_scale = grad_scale;
    if (flags & ~DRP_BATCH_REUSE_AA_RECORDS) return bfail("batch: unknown flags");
    drp::launch_batch_backward(a, workspace, L, (flags & DRP_BATCH_REUSE_AA_RECORDS) != 0,
                               static_cast<cudaStream_t>(stream));
    return drp_check_launch("drp_batch_backward");
}
