// interp.cu -- attribute interpolation forward/backward.
//
// Full-screen form replaces dr.interpolate (diffrp/rendering/interpolator.py:83);
// the sparse form replaces the torch gather + FMA of the stencil-masked
// interpolator (diffrp/rendering/interpolator.py:32-48, 87-97).  Both evaluate
//     out = fma(a0 - a2, u, fma(a1 - a2, v, a2))
// in that order (interpolator.py:45), one thread per pixel, with 128-bit
// vectorised attribute gathers and stores when the channel count is a multiple
// of four.  The backward scatters attribute gradients with float4 atomics
// after a warp-segmented reduction over runs of pixels that share a triangle, or,
// in larger launches, by columns of pixels (walk.cuh).
#include <algorithm>

#include "drp_common.cuh"
#include "drp_internal.h"
#include "walk.cuh"

namespace drp {

__device__ __forceinline__ float4 lerp_attr4(const float4& a0, const float4& a1, const float4& a2, float u, float v) {
    float4 o;
    o.x = fmaf(a0.x - a2.x, u, fmaf(a1.x - a2.x, v, a2.x));
    o.y = fmaf(a0.y - a2.y, u, fmaf(a1.y - a2.y, v, a2.y));
    o.z = fmaf(a0.z - a2.z, u, fmaf(a1.z - a2.z, v, a2.z));
    o.w = fmaf(a0.w - a2.w, u, fmaf(a1.w - a2.w, v, a2.w));
    return o;
}

__global__ void __launch_bounds__(256) interp_fwd_kernel(InterpArgs a) {
    const long long npix_view = (long long)a.H * a.W;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.B * npix_view) return;
    const int b = (int)(i / npix_view);
    const float4 r = reinterpret_cast<const float4*>(a.rast)[i];
    int j0 = 0, j1 = 0, j2 = 0;
    const int t = checked_tri(r.w, a.tri, a.num_triangles, a.num_vertices, j0, j1, j2);
    const int C = a.C;
    float* o = a.out + i * C;
    float* dd = a.da ? a.da + i * 2 * a.nd : nullptr;
    if (t < 0) {
        if ((C & 3) == 0) {
            for (int c = 0; c < C; c += 4) *reinterpret_cast<float4*>(o + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            for (int c = 0; c < C; ++c) o[c] = 0.f;
        }
        if (dd)
            for (int c = 0; c < 2 * a.nd; ++c) dd[c] = 0.f;
        return;
    }
    const float* A = a.attr + (long long)b * a.attr_view_stride;
    const long long i0 = j0, i1 = j1, i2 = j2;
    const float* a0 = A + i0 * C;
    const float* a1 = A + i1 * C;
    const float* a2 = A + i2 * C;
    const float u = r.x, v = r.y;
    if ((C & 3) == 0) {
        for (int c = 0; c < C; c += 4) {
            const float4 x0 = __ldg(reinterpret_cast<const float4*>(a0 + c));
            const float4 x1 = __ldg(reinterpret_cast<const float4*>(a1 + c));
            const float4 x2 = __ldg(reinterpret_cast<const float4*>(a2 + c));
            *reinterpret_cast<float4*>(o + c) = lerp_attr4(x0, x1, x2, u, v);
        }
    } else {
        for (int c = 0; c < C; ++c) {
            const float x0 = __ldg(a0 + c), x1 = __ldg(a1 + c), x2 = __ldg(a2 + c);
            o[c] = fmaf(x0 - x2, u, fmaf(x1 - x2, v, x2));
        }
    }
    if (dd) {
        const float4 db = reinterpret_cast<const float4*>(a.rast_db)[i];
        for (int k = 0; k < a.nd; ++k) {
            const int c = a.diff_idx[k];
            const float e0 = a0[c] - a2[c], e1 = a1[c] - a2[c];
            dd[2 * k + 0] = fmaf(e0, db.x, e1 * db.z);
            dd[2 * k + 1] = fmaf(e0, db.y, e1 * db.w);
        }
    }
}

__global__ void __launch_bounds__(256) interp_bwd_kernel(InterpArgs a) {
    const long long npix_view = (long long)a.H * a.W;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = i < (long long)a.B * npix_view;
    const int b = in ? (int)(i / npix_view) : 0;
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (in) r = reinterpret_cast<const float4*>(a.rast)[i];
    int j0 = 0, j1 = 0, j2 = 0;
    const int t = in ? checked_tri(r.w, a.tri, a.num_triangles, a.num_vertices, j0, j1, j2) : -1;
    const int C = a.C;
    const float* A = a.attr + (long long)b * a.attr_view_stride;
    float* G = a.grad_attr + (long long)b * a.attr_view_stride;
    const long long i0 = j0, i1 = j1, i2 = j2;
    const float u = r.x, v = r.y, w = 1.0f - u - v;
    const float* g = a.grad_out + (in ? i : 0) * C;
    float4 db = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* gdd = nullptr;
    if (t >= 0 && a.nd > 0 && a.grad_da) {
        db = reinterpret_cast<const float4*>(a.rast_db)[i];
        gdd = a.grad_da + i * 2 * a.nd;
    }
    const long long key = (t >= 0) ? (a.attr_view_stride ? (((long long)b << 32) | (long long)t) : (long long)t)
                                   : (long long)(-1 - lane_id());
    const Seg seg = seg_setup(key);
    float gu = 0.f, gv = 0.f;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
    for (int c0 = 0; c0 < C; c0 += 4) {
        float val[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) val[k] = 0.f;
        if (t >= 0) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c = c0 + k;
                if (c < C) {
                    const float gc = g[c];
                    float w0 = gc * u, w1 = gc * v, w2 = gc * w;
                    const float x0 = A[i0 * C + c], x1 = A[i1 * C + c], x2 = A[i2 * C + c];
                    gu = fmaf(gc, x0 - x2, gu);
                    gv = fmaf(gc, x1 - x2, gv);
                    if (gdd) {
                        for (int q = 0; q < a.nd; ++q) {
                            if (a.diff_idx[q] != c) continue;
                            const float gx = gdd[2 * q], gy = gdd[2 * q + 1];
                            const float d0 = fmaf(gx, db.x, gy * db.y), d1 = fmaf(gx, db.z, gy * db.w);
                            w0 += d0;
                            w1 += d1;
                            w2 -= d0 + d1;
                            s0 = fmaf(gx, x0 - x2, s0);
                            s1 = fmaf(gy, x0 - x2, s1);
                            s2 = fmaf(gx, x1 - x2, s2);
                            s3 = fmaf(gy, x1 - x2, s3);
                        }
                    }
                    val[k] = w0;
                    val[4 + k] = w1;
                    val[8 + k] = w2;
                }
            }
        }
        seg_reduce<12>(seg, val);
        if (t >= 0 && seg.head) {
            if ((C & 3) == 0) {
                atomic_add4(reinterpret_cast<float4*>(G + i0 * C + c0), make_float4(val[0], val[1], val[2], val[3]));
                atomic_add4(reinterpret_cast<float4*>(G + i1 * C + c0), make_float4(val[4], val[5], val[6], val[7]));
                atomic_add4(reinterpret_cast<float4*>(G + i2 * C + c0), make_float4(val[8], val[9], val[10], val[11]));
            } else {
                for (int k = 0; k < 4 && c0 + k < C; ++k) {
                    atomicAdd(G + i0 * C + c0 + k, val[k]);
                    atomicAdd(G + i1 * C + c0 + k, val[4 + k]);
                    atomicAdd(G + i2 * C + c0 + k, val[8 + k]);
                }
            }
        }
    }
    if (in) {
        if (a.grad_rast) reinterpret_cast<float4*>(a.grad_rast)[i] = make_float4(gu, gv, 0.f, 0.f);
        if (a.grad_db) reinterpret_cast<float4*>(a.grad_db)[i] = make_float4(s0, s1, s2, s3);
    }
}

// Backward of larger launches, by columns (walk.cuh): a warp takes 32 columns x
// a few rows of one view and up to 4 NG channels from c0 on; more channels
// are further walks over the same strip, which add to the first one's grad_rast
// and grad_db.  Rast rows and output gradients come by asynchronous copies two
// rows ahead, the next row's vertex indices one row ahead; the differences of
// the attributes stay in registers while the column is in its triangle.  DA:
// with gradients of the screen-space derivatives.  VEC: rows of 16-byte units.
// What bounds it: the latency of a strip's rows at 16 warps per SM, and the
// atomics.  4.8M pixels x 8 channels: 90 instead of 126 us; 4.2M x 5 with two
// derivatives: 147 instead of 202.
constexpr int kInterpStages = 3;
template <int NG, bool DA>
struct InterpWalkShared {
    WalkRows<3 * NG> rows;
    float4 rast[kInterpStages][32], db[DA ? kInterpStages : 1][32];
    float4 g[kInterpStages][NG][32];
};

// The next place from q on where channel c is listed, or -1.
__device__ __forceinline__ int next_diff(const InterpArgs& a, int q, int c) {
    for (; q < a.nd; ++q)
        if (a.diff_idx[q] == c) return q;
    return -1;
}

template <int NG, bool VEC, bool DA>
__device__ __forceinline__ void interp_walk(const InterpArgs& a, const WalkStrip& s, int c0,
                                            InterpWalkShared<NG, DA>& sh) {
    constexpr int Q = 3 * NG;
    const int lane = threadIdx.x & 31, x = s.x0 + lane;
    const int W = a.W, C = a.C, cn = VEC ? 4 * NG : min(C - c0, 4 * NG);
    const bool in = x < W, more = c0 > 0;
    const long long view = (long long)s.b * a.H * W;
    const float4* R = reinterpret_cast<const float4*>(a.rast) + view;
    const float* G = a.grad_out + view * C + c0;
    const float* A = a.attr + (long long)s.b * a.attr_view_stride + c0;
    float* GA = a.grad_attr + (long long)s.b * a.attr_view_stride + c0;
    // the column's triangle: attribute differences to its third vertex, sums
    // (vertex i, channels 2 k, 2 k + 1), vertices
    f32x2 d0[2 * NG], d1[2 * NG], acc[3][2 * NG];
    int cur = -1, j0 = 0, j1 = 0, j2 = 0, n = 0;
#pragma unroll
    for (int k = 0; k < 2 * NG; ++k) {
        d0[k] = d1[k] = 0ull;
#pragma unroll
        for (int i = 0; i < 3; ++i) acc[i][k] = 0ull;
    }
    const auto leave = [&](float* row) {
        f32x2* d = reinterpret_cast<f32x2*>(row);
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int i = 0; i < 3; ++i)
                *reinterpret_cast<ulonglong2*>(d + 6 * g + 2 * i) = make_ulonglong2(acc[i][2 * g], acc[i][2 * g + 1]);
        *reinterpret_cast<int4*>(row + 4 * Q) = make_int4(j0, j1, j2, 0);
    };
    const auto add = [&](const float* row, int quad, const float4& v) {
        const int cg = 4 * (quad / 3);
        float* d = GA + (long long)__float_as_int(row[4 * Q + quad % 3]) * C + cg;
        if (VEC) {
            atomic_add4(reinterpret_cast<float4*>(d), v);
        } else {
            if (cg < cn) atomicAdd(d, v.x);
            if (cg + 1 < cn) atomicAdd(d + 1, v.y);
            if (cg + 2 < cn) atomicAdd(d + 2, v.z);
            if (cg + 3 < cn) atomicAdd(d + 3, v.w);
        }
    };
    const auto request = [&](int y) {
        if (in && y < s.y1) {
            const int st = (y - s.y0) % kInterpStages;
            const long long p = (long long)y * W + x;
            cp_async<16>(&sh.rast[st][lane], R + p);
            if (DA) cp_async<16>(&sh.db[DA ? st : 0][lane], reinterpret_cast<const float4*>(a.rast_db) + view + p);
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                float* d = reinterpret_cast<float*>(&sh.g[st][g][lane]);
                if (VEC) {
                    cp_async<16>(d, G + p * C + 4 * g);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (4 * g + k < cn) cp_async<4>(d + k, G + p * C + 4 * g + k);
                }
            }
        }
        cp_async_commit();
    };
    if (!VEC) {  // channels past the last stay zero
#pragma unroll
        for (int k = 0; k < kInterpStages; ++k)
#pragma unroll
            for (int c = 0; c < 4 * NG; ++c)
                if (c >= cn) reinterpret_cast<float*>(&sh.g[k][c >> 2][lane])[c & 3] = 0.f;
    }
    // DA: where each channel is listed (first place), and whether one is twice
    int first[4 * NG];
    bool twice = false;
    if (DA) {
#pragma unroll
        for (int c = 0; c < 4 * NG; ++c) {
            first[c] = c < cn ? next_diff(a, 0, c0 + c) : -1;
            if (first[c] >= 0) twice = twice || next_diff(a, first[c] + 1, c0 + c) >= 0;
        }
    }
    request(s.y0);
    request(s.y0 + 1);
    cp_async_wait<1>();  // row y0 (this lane's part, as below)
    int i0 = 0, i1 = 0, i2 = 0;
    int t = in ? checked_tri(sh.rast[0][lane].w, a.tri, a.num_triangles, a.num_vertices, i0, i1, i2) : -1;
    int st = 0;
#pragma unroll 1
    for (int y = s.y0; y < s.y1; ++y) {
        request(y + 2);
        cp_async_wait<1>();  // row y + 1
        const int stn = st + 1 == kInterpStages ? 0 : st + 1;
        int n0 = i0, n1 = i1, n2 = i2, tn = -1;
        if (in && y + 1 < s.y1) {
            const float id = sh.rast[stn][lane].w;
            tn = t;
            if (id != sh.rast[st][lane].w) tn = checked_tri(id, a.tri, a.num_triangles, a.num_vertices, n0, n1, n2);
        }
        const bool live = t >= 0, enter = live && t != cur;
        walk_leave<Q>(sh.rows, n, enter && cur >= 0, leave, add);
        if (enter) {
            cur = t;
            j0 = i0;
            j1 = i1;
            j2 = i2;
#pragma unroll
            for (int k = 0; k < 2 * NG; ++k)
#pragma unroll
                for (int i = 0; i < 3; ++i) acc[i][k] = 0ull;
            const float *a0 = A + (long long)i0 * C, *a1 = A + (long long)i1 * C, *a2 = A + (long long)i2 * C;
            float x0[4 * NG], x1[4 * NG], x2[4 * NG];
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                load4<VEC>(a0 + 4 * g, cn - 4 * g, x0 + 4 * g);
                load4<VEC>(a1 + 4 * g, cn - 4 * g, x1 + 4 * g);
                load4<VEC>(a2 + 4 * g, cn - 4 * g, x2 + 4 * g);
            }
#pragma unroll
            for (int k = 0; k < 2 * NG; ++k) {
                d0[k] = pack2(x0[2 * k] - x2[2 * k], x0[2 * k + 1] - x2[2 * k + 1]);
                d1[k] = pack2(x1[2 * k] - x2[2 * k], x1[2 * k + 1] - x2[2 * k + 1]);
            }
        }
        float gu = 0.f, gv = 0.f;
        float4 gdb = make_float4(0.f, 0.f, 0.f, 0.f);
        const long long p = view + (long long)y * W + x;
        if (live) {
            const float4 r4 = sh.rast[st][lane];
            const float u = r4.x, v = r4.y, w = 1.0f - u - v;
            const f32x2 bb[3] = {pack2(u, u), pack2(v, v), pack2(w, w)};
#pragma unroll
            for (int k = 0; k < 2 * NG; ++k) {
                const ulonglong2 gq = *reinterpret_cast<const ulonglong2*>(&sh.g[st][k >> 1][lane]);
                const f32x2 gg = (k & 1) ? gq.y : gq.x;
                gu = fmaf(hi2(gg), hi2(d0[k]), fmaf(lo2(gg), lo2(d0[k]), gu));
                gv = fmaf(hi2(gg), hi2(d1[k]), fmaf(lo2(gg), lo2(d1[k]), gv));
#pragma unroll
                for (int i = 0; i < 3; ++i) acc[i][k] = fma2(gg, bb[i], acc[i][k]);
            }
            if (DA) {
                const float4 db = sh.db[DA ? st : 0][lane];
                const float* gdd = a.grad_da + p * 2 * a.nd;
#pragma unroll
                for (int c = 0; c < 4 * NG; ++c) {
                    const int k = c >> 1;
                    const bool hi = c & 1;
                    for (int q = first[c]; q >= 0; q = twice ? next_diff(a, q + 1, c0 + c) : -1) {
                        const float gx = gdd[2 * q], gy = gdd[2 * q + 1];
                        const float e0 = fmaf(gx, db.x, gy * db.y), e1 = fmaf(gx, db.z, gy * db.w);
                        const float f0 = hi ? hi2(d0[k]) : lo2(d0[k]), f1 = hi ? hi2(d1[k]) : lo2(d1[k]);
                        const float e[3] = {e0, e1, -(e0 + e1)};
#pragma unroll
                        for (int i = 0; i < 3; ++i)
                            acc[i][k] = hi ? pack2(lo2(acc[i][k]), hi2(acc[i][k]) + e[i])
                                           : pack2(lo2(acc[i][k]) + e[i], hi2(acc[i][k]));
                        gdb.x = fmaf(gx, f0, gdb.x);
                        gdb.y = fmaf(gy, f0, gdb.y);
                        gdb.z = fmaf(gx, f1, gdb.z);
                        gdb.w = fmaf(gy, f1, gdb.w);
                    }
                }
            }
        }
        if (in && a.grad_rast) {
            float4* o = reinterpret_cast<float4*>(a.grad_rast) + p;
            if (more) {
                const float4 o4 = *o;
                gu += o4.x;
                gv += o4.y;
            }
            *o = make_float4(gu, gv, 0.f, 0.f);
        }
        if (in && a.grad_db) {
            float4* o = reinterpret_cast<float4*>(a.grad_db) + p;
            if (more) {
                const float4 o4 = *o;
                gdb = make_float4(gdb.x + o4.x, gdb.y + o4.y, gdb.z + o4.z, gdb.w + o4.w);
            }
            *o = gdb;
        }
        t = tn;
        i0 = n0;
        i1 = n1;
        i2 = n2;
        st = stn;
    }
    walk_leave<Q>(sh.rows, n, cur >= 0, leave, add);
    if (n) walk_drain<Q>(sh.rows, n, add);
}

template <bool DA>
__global__ void __launch_bounds__(32 * kWalkWarps, 16 / kWalkWarps) interp_bwd_walk_kernel(InterpArgs a, int rows) {
    __shared__ union {
        InterpWalkShared<1, DA> one;
        InterpWalkShared<2, DA> two;
    } sh[kWalkWarps];
    WalkStrip s;
    if (!walk_strip(a.B, a.H, a.W, rows, s)) return;
    const int warp = threadIdx.x >> 5;
    const bool vec = (a.C & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.attr) | reinterpret_cast<uintptr_t>(a.grad_attr) |
                                         reinterpret_cast<uintptr_t>(a.grad_out)) & 15) == 0;
    for (int c0 = 0; c0 < a.C; c0 += 8) {
        if (vec && a.C - c0 >= 8) interp_walk<2, true, DA>(a, s, c0, sh[warp].two);
        else if (vec) interp_walk<1, true, DA>(a, s, c0, sh[warp].one);
        else if (a.C - c0 > 4) interp_walk<2, false, DA>(a, s, c0, sh[warp].two);
        else interp_walk<1, false, DA>(a, s, c0, sh[warp].one);
        __syncwarp();
    }
}

// Sparse form: vi (N, 4) rast rows, tri_idx (N, 3) int64 vertex indices.
__global__ void __launch_bounds__(256) interp_sparse_fwd_kernel(SparseInterpArgs a) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= a.N) return;
    const int C = a.C;
    const float4 r = reinterpret_cast<const float4*>(a.vi)[n];
    const long long i0 = a.tri_idx[3 * n], i1 = a.tri_idx[3 * n + 1], i2 = a.tri_idx[3 * n + 2];
    float* o = a.out + n * C;
    if (i0 < 0 || i1 < 0 || i2 < 0 || i0 >= a.V || i1 >= a.V || i2 >= a.V) {
        for (int c = 0; c < C; ++c) o[c] = __int_as_float(0x7fc00000);
        return;
    }
    const float* a0 = a.vb + i0 * C;
    const float* a1 = a.vb + i1 * C;
    const float* a2 = a.vb + i2 * C;
    if ((C & 3) == 0) {
        for (int c = 0; c < C; c += 4) {
            const float4 x0 = __ldg(reinterpret_cast<const float4*>(a0 + c));
            const float4 x1 = __ldg(reinterpret_cast<const float4*>(a1 + c));
            const float4 x2 = __ldg(reinterpret_cast<const float4*>(a2 + c));
            *reinterpret_cast<float4*>(o + c) = lerp_attr4(x0, x1, x2, r.x, r.y);
        }
    } else {
        for (int c = 0; c < C; ++c) {
            const float x0 = __ldg(a0 + c), x1 = __ldg(a1 + c), x2 = __ldg(a2 + c);
            o[c] = fmaf(x0 - x2, r.x, fmaf(x1 - x2, r.y, x2));
        }
    }
}

__global__ void __launch_bounds__(256) interp_sparse_bwd_kernel(SparseInterpArgs a) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool in = n < a.N;
    const int C = a.C;
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    long long i0 = 0, i1 = 0, i2 = 0;
    if (in) {
        r = reinterpret_cast<const float4*>(a.vi)[n];
        i0 = a.tri_idx[3 * n];
        i1 = a.tri_idx[3 * n + 1];
        i2 = a.tri_idx[3 * n + 2];
        if (i0 < 0 || i1 < 0 || i2 < 0 || i0 >= a.V || i1 >= a.V || i2 >= a.V) {
            in = false;
            i0 = i1 = i2 = 0;
            if (a.grad_vi) reinterpret_cast<float4*>(a.grad_vi)[n] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    // Runs keyed by the first vertex index of the row's triangle.
    const long long key = in ? (i0 ^ (i1 << 21) ^ (i2 << 42)) : (long long)(-1 - lane_id());
    const Seg seg = seg_setup(key);
    const float u = r.x, v = r.y, w = 1.0f - u - v;
    float gu = 0.f, gv = 0.f;
    for (int c0 = 0; c0 < C; c0 += 4) {
        float val[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) val[k] = 0.f;
        if (in) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c = c0 + k;
                if (c < C) {
                    const float gc = a.grad_out[n * C + c];
                    const float x0 = a.vb[i0 * C + c], x1 = a.vb[i1 * C + c], x2 = a.vb[i2 * C + c];
                    val[k] = gc * u;
                    val[4 + k] = gc * v;
                    val[8 + k] = gc * w;
                    gu = fmaf(gc, x0 - x2, gu);
                    gv = fmaf(gc, x1 - x2, gv);
                }
            }
        }
        seg_reduce<12>(seg, val);
        if (in && seg.head) {
            for (int k = 0; k < 4 && c0 + k < C; ++k) {
                atomicAdd(a.grad_vb + i0 * C + c0 + k, val[k]);
                atomicAdd(a.grad_vb + i1 * C + c0 + k, val[4 + k]);
                atomicAdd(a.grad_vb + i2 * C + c0 + k, val[8 + k]);
            }
        }
    }
    if (in && a.grad_vi) reinterpret_cast<float4*>(a.grad_vi)[n] = make_float4(gu, gv, 0.f, 0.f);
}

int launch_interp_fwd(const InterpArgs& a, cudaStream_t s) {
    const long long n = (long long)a.B * a.H * a.W;
    if (n == 0) return 0;
    interp_fwd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    drp_note_launch();
    return 0;
}

// Pixels from which the backward goes by columns.  A strip is a long chain for
// one warp, and the old kernel's cost is the shuffles and, where vectors do not
// fit the rows, its scalar atomics: per channel count, us by pixels against by
// columns, on the mesh that gains least: 3 channels at 700 x 700 16.9 / 14.9;
// 4 at 2M pixels 43.2 / 41.5 (1M 22.3 / 23.4); 8 at 1M 32.0 / 29.4; 10 at
// 700 x 700 38.6 / 33.5; 16 38.3 / 34.5; 1 at 4.2M 76.4 / 75.6 (2M 37.3 / 43.3).
// 12 (a walk of eight and one of four) stays: 4.2M 155 / 170.  With derivatives:
// 5 of 2 at 4.2M 194 / 165 (1M 52.6 / 53.7), 8 of 2 171 / 160, 4 of 4 134 / 143.
// Up to four channels or with derivatives a pixel costs the walk little more than
// a triangle that the column leaves, so meshes of triangles of a few pixels stay
// by pixels too (kWalkPixelsPerPrim; 318k triangles a view, six views of 800 x
// 1000: 1 channel 86 by pixels against 115, 2 100 / 121, 4 100 / 119, 3 of 2
// derivatives 148 / 176; 1440 x 1080, five pixels a triangle: 3 49 / 52).
constexpr long long kWalkPixelsPerPrim = 6;
static long long interp_walk_pixels(int C, bool da, long long prims) {
    const long long never = 1ll << 62;
    if (C % 8 == 4 && (C > 4 || da)) return never;
    const long long few = C <= 4 || da ? kWalkPixelsPerPrim * prims : 0;
    if (da) return C < 3 ? never : std::max(1ll << 22, few);
    if (C <= 2) return std::max(1ll << 22, few);
    return std::max(C == 4 ? 1ll << 21 : (C == 8 ? 1ll << 20 : 1ll << 19), few);
}

// Rows per warp: from 2^20 pixels on 16, for fewer sums to add (3 channels, a mesh
// of 642 vertices at 4.2M pixels: 128 -> 86 us, its atomics collide); two walks
// over a strip of 8 find its rast rows in cache.
static int interp_walk_rows(int C, long long n) { return n >= 1ll << 20 && C <= 8 ? 16 : 8; }

int launch_interp_bwd(const InterpArgs& a, cudaStream_t s) {
    const long long n = (long long)a.B * a.H * a.W;
    if (n == 0) return 0;
    const bool da = a.nd > 0 && a.grad_da;
    const int rows = interp_walk_rows(a.C, n);
    if (n < interp_walk_pixels(a.C, da, a.num_triangles * a.B))
        interp_bwd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    else if (da)
        interp_bwd_walk_kernel<true><<<walk_blocks(a.B, a.H, a.W, rows), 32 * kWalkWarps, 0, s>>>(a, rows);
    else
        interp_bwd_walk_kernel<false><<<walk_blocks(a.B, a.H, a.W, rows), 32 * kWalkWarps, 0, s>>>(a, rows);
    drp_note_launch();
    return 0;
}

int launch_interp_sparse_fwd(const SparseInterpArgs& a, cudaStream_t s) {
    if (a.N == 0) return 0;
    interp_sparse_fwd_kernel<<<(unsigned)((a.N + 255) / 256), 256, 0, s>>>(a);
    drp_note_launch();
    return 0;
}

int launch_interp_sparse_bwd(const SparseInterpArgs& a, cudaStream_t s) {
    if (a.N == 0) return 0;
    interp_sparse_bwd_kernel<<<(unsigned)((a.N + 255) / 256), 256, 0, s>>>(a);
    drp_note_launch();
    return 0;
}

}  // namespace drp
