// kv_rc.cu -- RC family: the reference projector pair reproduced on sm_103a.
//
// Forward: source/modules/reconstruction/Projector.cu:227-372 (kernel) with
// FindProjectionAlphas_d Projector.cu:45-223.  Each ray's plane-crossing
// parameters form three ascending arithmetic sequences (x, y and z planes,
// each generated by repeated addition exactly as the reference fills its
// list) plus the entries the reference leaves at 1.0.  The reference sorts
// that list with an O(n^2) selection sort in 8 KB of thread-local memory;
// here the sorted order is produced by a four-way merge of the sequences in
// registers, which yields the same sorted values.  The segment midpoint is
// computed in double by the reference (Projector.cu:350-354); here it is
// evaluated in float and redone in double only when the float result is an
// integer, so the truncated index is the same.
//
// Backprojector: Projector.cu:376-785, one thread per voxel, an 11x11 window
// of pixel rays per view, weights normalised by their sum.  The x-plane
// parameters of the window's columns are computed once per view instead of
// once per pixel (same values, same operations), and the window is first cut
// to the pixels whose rays can meet the voxel: the others have an empty
// intersection and add nothing.  All 11 x 11 pixels of one voxel a thread, with
// some 50 divisions, took 5.4 ms on 256 x 256 x 64 voxels and 15 views; the cut
// window 1.5 ms; the column intervals shared by four rows of a thread and the
// row intervals by a warp, the view's constants by a block: 0.54 ms.
//
// This translation unit is compiled with -fmad=false: no multiply-add is
// fused, matching the reference kernel source compiled for the host, against
// which the results are bit-identical.
#include "kv_internal.h"

namespace {

struct RcGeom {
    int nx, ny, nz, nu, nv, n_views;
    float dx, dy, dz, du, dv;
};

__device__ __forceinline__ bool rc_sup_eq(float a, float b) {
    const float d = a - b;
    return a > b || (d < 0.0000001F && d > -0.0000001F);
}

// (int)((double)base + (double)c * (double)d), Projector.cu:352-354.  v is the exact sum rounded to float once (the
// product is exact in double): rounding never carries it across an integer, so v and the double sum have the same
// integer part unless v is an integer itself.  Only then is the sum formed in double, out of line: inlined, the
// compiler ran the double arithmetic for every index and selected afterwards, and the FP64 pipe bounded the kernel
// (15 views of 512 x 512 through 256 x 256 x 64 voxels: 3.9 -> 0.53 ms).  A NaN (a source or detector so far off that
// its position in voxels overflows) takes the double path too, where it becomes no voxel's index; as a float it would
// convert to 0.
__device__ __noinline__ int rc_index_double(float base, float c, float d) {
    return (int)((double)base + (double)c * (double)d);
}

__device__ __forceinline__ int rc_index(float base, float c, float d) {
    const float v = fmaf(c, d, base);
    const float r = rintf(v);
    return v < r || v > r ? (int)v : rc_index_double(base, c, d);
}

// Window pixels [q0, q1] cut to those whose ray can meet the voxel: a ray's parameter lies in [mn, mx] there (the
// voxel's z planes), so its component dr obeys f - s <= dr * a <= f + 1 - s for some a of them.  A margin of 0.05 pixel
// and 1e-5 of the position covers the rounding of both evaluations (a few 1e-7 of the position); a pixel outside has
// an empty interval in the full evaluation too and adds nothing.  o, d: detector origin and pitch in mm, dv: voxel
// pitch, in the window's own units.
__device__ __forceinline__ void rc_cut(int &q0, int &q1, float f, float s, float mn, float mx, float o, float d,
                                       float dv) {
    if (!(mn > 1e-3f && mx < 1e3f)) return;   // a plane at or behind the source: the whole window
    const float a = f - s, b = a + 1.F, in = 1.F / mn, ix = 1.F / mx;
    const float lo = fminf(fminf(a * in, a * ix), fminf(b * in, b * ix));
    const float hi = fmaxf(fmaxf(a * in, a * ix), fmaxf(b * in, b * ix));
    const float plo = ((lo + s) * dv - o) / d - 0.5F, phi = ((hi + s) * dv - o) / d - 0.5F;
    const float m = 0.05F + 1e-5F * (fabsf(plo) + fabsf(phi) + fabsf(o / d) + fabsf(s * dv / d));
    if (!(plo > -1e6f && phi < 1e6f)) return;
    q0 = max(q0, (int)ceilf(plo - m));
    q1 = min(q1, (int)floorf(phi + m));
}

struct Seq {
    float val, step;
    int left;
};

template <int MODE>
__global__ void __launch_bounds__(128) rc_forward_kernel(RcGeom G, const float *__restrict__ src,
                                                         const float *__restrict__ org,
                                                         const float *__restrict__ vol,
                                                         const float *__restrict__ meas,
                                                         float *__restrict__ out, float relax) {
    const int u = blockIdx.x * 32 + threadIdx.x;
    const int v = blockIdx.y * blockDim.y + threadIdx.y;
    const int p = blockIdx.z;
    if (u >= G.nu || v >= G.nv) return;
    const size_t ray = ((size_t)p * G.nv + v) * G.nu + u;
    const float tol = 0.000001F;
    const int n[3] = {G.nx, G.ny, G.nz};
    float s[3], d[3], half[3];
    s[0] = src[3 * p] / G.dx;
    s[1] = src[3 * p + 1] / G.dy;
    s[2] = src[3 * p + 2] / G.dz;
    const float px = (org[3 * p] + ((float)u + 0.5F) * G.du) / G.dx;
    const float py = (org[3 * p + 1] + ((float)v + 0.5F) * G.dv) / G.dy;
    const float pz = org[3 * p + 2] / G.dz;
    d[0] = px - s[0];
    d[1] = py - s[1];
    d[2] = pz - s[2];
#pragma unroll
    for (int a = 0; a < 3; ++a) half[a] = (float)n[a] / 2.F;

    float mins[3], maxs[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float a1 = fabsf(d[a]) > tol ? (-half[a] - s[a]) / d[a] : 0.F;
        const float aN = fabsf(d[a]) > tol ? (half[a] - s[a]) / d[a] : 0.F;
        mins[a] = fminf(a1, aN);
        maxs[a] = fmaxf(a1, aN);
    }
    const float amin = fmaxf(fmaxf(0.F, mins[0]), fmaxf(mins[1], mins[2]));
    const float amax = fminf(fminf(1.F, maxs[0]), fminf(maxs[1], maxs[2]));
    float q = 0.F;
    if (!rc_sup_eq(amin, amax)) {
        Seq sq[3];
        int total = 3, filled = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float at_hi = d[a] > 0 ? amax : amin;
            const float at_lo = d[a] > 0 ? amin : amax;
            const float up = (half[a] + s[a]) + at_hi * d[a];
            const int mx = max(0, min(n[a] - 1, (int)up));
            const float dn = (half[a] - s[a]) - at_lo * d[a];
            const int mn = max(0, min(mx, n[a] - (int)dn));
            const int span = mx - mn;
            total += span;
            const int count = a < 2 ? span + 1 : (span >= 2 ? span - 1 : 1);
            if (fabsf(d[a]) > tol) {
                const float step = 1.F / d[a];
                const float plane = (float)(d[a] > 0 ? mn : mx);
                sq[a].val = step * ((-half[a] - s[a]) + plane);
                sq[a].step = fabsf(step);
                sq[a].left = count;
                filled += count;
            } else {
                sq[a].val = 0.F;
                sq[a].step = 0.F;
                sq[a].left = 0;
            }
        }
        int ones = total - filled;   // entries left at the fill value 1.0
        const float b0 = half[0] + s[0], b1 = half[1] + s[1], b2 = half[2] + s[2];
        const float d0 = d[0], d1 = d[1], d2 = d[2];
        // the three sequences as scalars (a dynamically indexed array would
        // live in local memory and every merge step would go through L1)
        float v0 = sq[0].val, v1 = sq[1].val, v2 = sq[2].val;
        const float st0 = sq[0].step, st1 = sq[1].step, st2 = sq[2].step;
        int l0 = sq[0].left, l1 = sq[1].left, l2 = sq[2].left;
        float acc = 0.F, wsum = 0.F;
        float prev = 0.F;
        for (int e = 0; e < total; ++e) {
            // pop the smallest head among x, y, z and the 1.0 entries
            float best = 3.402823466e38F;
            int which = 3;
            if (l0 > 0) { best = v0; which = 0; }
            if (l1 > 0 && v1 < best) { best = v1; which = 1; }
            if (l2 > 0 && v2 < best) { best = v2; which = 2; }
            if (ones > 0 && 1.0F < best) { best = 1.0F; which = 3; }
            if (which == 0) {
                v0 = v0 + st0;
                --l0;
            } else if (which == 1) {
                v1 = v1 + st1;
                --l1;
            } else if (which == 2) {
                v2 = v2 + st2;
                --l2;
            } else if (ones > 0) {
                --ones;
            }
            if (e > 0) {
                const float c = (best + prev) * 0.5F;
                const int ix = rc_index(b0, c, d0);
                const int iy = rc_index(b1, c, d1);
                const int iz = rc_index(b2, c, d2);
                const float w = best - prev;
                if (ix >= 0 && ix < G.nx && iy >= 0 && iy < G.ny && iz >= 0 && iz < G.nz && w > tol) {
                    const size_t idx = ((size_t)iz * G.ny + iy) * G.nx + ix;
                    wsum += w;
                    acc += w * __ldg(vol + idx);
                }
            }
            prev = best;
        }
        q = wsum > tol ? acc / wsum : 0.F;
    }
    if (MODE == RC_PLAIN) {
        out[ray] = q;
    } else if (MODE == RC_MLEM) {
        // Reconstructors.h:207-213: ratio where q != 0 (AlmostEqualRelative)
        out[ray] = q != 0.F ? relax * (meas[ray] / q) : q;
    } else {
        // Reconstructors.h:90-93
        out[ray] = relax * (meas[ray] - q);
    }
}

// Ray components of the detector columns and rows of every view, source to pixel in voxel units (the backprojector
// needs them for every voxel): tab[p][u] = x, then [p][v] = y.
__global__ void rc_table_kernel(RcGeom G, const float *__restrict__ src, const float *__restrict__ org,
                                float *__restrict__ tab) {
    const int p = blockIdx.x;
    const float ox = org[3 * p], sx = src[3 * p] / G.dx;
    for (int q = threadIdx.x; q < G.nu; q += blockDim.x)
        tab[(size_t)p * G.nu + q] = (ox + ((float)q + 0.5F) * G.du) / G.dx - sx;
    const float oy = org[3 * p + 1], sy = src[3 * p + 1] / G.dy;
    for (int q = threadIdx.x; q < G.nv; q += blockDim.x)
        tab[(size_t)G.n_views * G.nu + (size_t)p * G.nv + q] = (oy + ((float)q + 0.5F) * G.dv) / G.dy - sy;
}

// What of a view depends on the slice only, computed once per block.
struct RcView {
    float ox, oy, sx, sy, ofx, ofy, ex, ey, az, mnz, mxz, pad;
};

constexpr int kRcRows = 4;                 // voxel rows of a thread, 4 apart
constexpr int kRcFill = 32 / kRcRows;      // window rows of one voxel row computed side by side
constexpr int kRcViews = 64;               // views whose constants a block holds at a time

// Block = 32 columns x 16 rows of slice z (4 warps, warp w rows w, w + 4, w + 8, w + 12).  Per view a lane computes
// the parameter intervals of its column's window columns once for its four rows; those of the window rows, which are
// the same for the whole warp, are computed one (row, window row) a lane into shared memory.
template <int MODE>
__global__ void __launch_bounds__(128) rc_back_kernel(RcGeom G, const float *__restrict__ src,
                                                      const float *__restrict__ org, const float *__restrict__ tab,
                                                      const float *__restrict__ proj, float *__restrict__ vol, int z0) {
    __shared__ RcView views[kRcViews];
    __shared__ float2 ysh[4][kRcRows][12];
    const int lane = threadIdx.x, warp = threadIdx.y;
    const int x = blockIdx.x * 32 + lane, yw = blockIdx.y * 4 * kRcRows + warp;   // voxel rows yw + 4 r
    const int z = z0 + (int)blockIdx.z;   // slices z0 .. z0 + gridDim.z - 1
    const float tol = 0.000000000000000000000001F;
    const int semi = 5;
    const float vfx = (float)x - (float)G.nx / 2.F;
    const float vfz = (float)z - (float)G.nz / 2.F;
    const float mx = (float)semi * G.du / G.dx, my = (float)semi * G.dv / G.dy;
    const float *tabx = tab, *taby = tab + (size_t)G.n_views * G.nu;
    const int rf = lane / kRcFill, cf = lane % kRcFill;   // this lane fills window row cf (+ kRcFill f) of voxel row rf
    float acc[kRcRows], wsum[kRcRows];
#pragma unroll
    for (int r = 0; r < kRcRows; ++r) acc[r] = wsum[r] = 0.F;
    for (int pb = 0; pb < G.n_views; pb += kRcViews) {
        const int pn = min(kRcViews, G.n_views - pb);
        __syncthreads();
        for (int i = warp * 32 + lane; i < pn; i += 128) {
            const int p = pb + i;
            const float ox = org[3 * p], oy = org[3 * p + 1], oz = org[3 * p + 2];
            const float sx = src[3 * p] / G.dx, sy = src[3 * p + 1] / G.dy, sz = src[3 * p + 2] / G.dz;
            const float ofz = oz / G.dz, rz = (vfz + 0.5F) - sz;
            const float dzr = oz / G.dz - sz;
            const float a1z = fabsf(dzr) > tol ? (vfz - sz) / dzr : 0.F;
            const float a2z = fabsf(dzr) > tol ? (vfz + 1.F - sz) / dzr : 0.F;
            views[i] = RcView{ox, oy, sx, sy, ox / G.dx, oy / G.dy, (ox + (float)G.nu * G.du) / G.dx,
                              (oy + (float)G.nv * G.dv) / G.dy, fabsf(rz) > tol ? (ofz - sz) / rz : 0.F,
                              fminf(a1z, a2z), fmaxf(a1z, a2z), 0.F};
        }
        __syncthreads();
        for (int i = 0; i < pn; ++i) {
            const int p = pb + i;
            const RcView V = views[i];
            // window columns of voxel column x
            const float hx = V.sx + ((vfx + 0.5F) - V.sx) * V.az;
            int x0 = 0, x1 = -1;
            if (x < G.nx && hx > V.ofx - mx && hx < V.ex + mx) {
                const int pxl = (int)((hx - V.ofx) * G.dx / G.du);
                x0 = max(0, min(G.nu - 1, pxl - semi));
                x1 = max(0, min(G.nu - 1, pxl + semi));
                rc_cut(x0, x1, vfx, V.sx, V.mnz, V.mxz, V.ox, G.du, G.dx);
            }
            // window rows of this lane's fill row
            const int yf = yw + 4 * rf;
            const float vfy = (float)yf - (float)G.ny / 2.F;
            const float hy = V.sy + ((vfy + 0.5F) - V.sy) * V.az;
            int y0 = 0, y1 = -1;
            if (yf < G.ny && hy > V.ofy - my && hy < V.ey + my) {
                const int pyl = (int)((hy - V.ofy) * G.dy / G.dv);
                y0 = max(0, min(G.nv - 1, pyl - semi));
                y1 = max(0, min(G.nv - 1, pyl + semi));
                rc_cut(y0, y1, vfy, V.sy, V.mnz, V.mxz, V.oy, G.dv, G.dy);
            }
            const int nyf = max(0, y1 - y0 + 1);   // at most 11
            const int ncol = x1 - x0 + 1;
            const int nymax = __reduce_max_sync(0xffffffffu, nyf);
            if (nymax == 0 || __reduce_max_sync(0xffffffffu, ncol) <= 0) continue;   // warp-uniform
            __syncwarp();
            for (int f = 0; f * kRcFill < nymax; ++f) {
                const int c = f * kRcFill + cf;
                if (c < nyf) {
                    const float dyr = __ldg(taby + (size_t)p * G.nv + y0 + c);
                    const float a1y = fabsf(dyr) > tol ? (vfy - V.sy) / dyr : 0.F;
                    const float a2y = fabsf(dyr) > tol ? (vfy + 1.F - V.sy) / dyr : 0.F;
                    ysh[warp][rf][c] = make_float2(fmaxf(fminf(a1y, a2y), V.mnz), fminf(fmaxf(a1y, a2y), V.mxz));
                }
            }
            __syncwarp();
            // x parameters of the window columns (at most 11; the cut leaves about four)
            float cmn[11], cmx[11];
#pragma unroll
            for (int c = 0; c < 11; ++c) {
                if (c >= ncol) break;
                const float dxr = __ldg(tabx + (size_t)p * G.nu + x0 + c);
                const float a1x = fabsf(dxr) > tol ? (vfx - V.sx) / dxr : 0.F;
                const float a2x = fabsf(dxr) > tol ? (vfx + 1.F - V.sx) / dxr : 0.F;
                cmn[c] = fmaxf(0.F, fminf(a1x, a2x));
                cmx[c] = fminf(1.F, fmaxf(a1x, a2x));
            }
            const float *pv = proj + (size_t)p * G.nu * G.nv + x0;
#pragma unroll
            for (int r = 0; r < kRcRows; ++r) {
                const int ny = __shfl_sync(0xffffffffu, nyf, r * kRcFill);
                const float *row = pv + (size_t)__shfl_sync(0xffffffffu, y0, r * kRcFill) * G.nu;
                for (int q = 0; q < ny; ++q, row += G.nu) {
                    const float2 yi = ysh[warp][r][q];
#pragma unroll
                    for (int c = 0; c < 11; ++c) {
                        if (c >= ncol) break;
                        const float lo = fmaxf(cmn[c], yi.x);
                        const float hi = fminf(cmx[c], yi.y);
                        const float w = hi - lo;
                        if (w > tol) {   // and so hi > lo, the reference's first test
                            wsum[r] += w;
                            acc[r] += w * __ldg(row + c);
                        }
                    }
                }
            }
        }
    }
    if (x >= G.nx) return;
#pragma unroll
    for (int r = 0; r < kRcRows; ++r) {
        const int y = yw + 4 * r;
        if (y >= G.ny) continue;
        const float b = wsum[r] > tol ? acc[r] / wsum[r] : 0.F;
        const size_t idx = ((size_t)z * G.ny + y) * G.nx + x;
        if (MODE == RC_PLAIN) vol[idx] = b;
        else if (MODE == RC_MLEM) vol[idx] = vol[idx] * b;     // Reconstructors.h:238-241
        else vol[idx] = vol[idx] + b;                          // Reconstructors.h:118-121
    }
}

// Elementwise ratio step of recons::MLEM / recons::ART on a forward result q,
// the same float operations as the fused epilogue of rc_forward_kernel.
__global__ void rc_ratio_kernel(int mode, const float *__restrict__ p, float *__restrict__ q, size_t n,
                                float relax) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float qi = q[i];
        q[i] = mode == RC_MLEM ? (qi != 0.F ? relax * (p[i] / qi) : qi) : relax * (p[i] - qi);
    }
}

RcGeom rcgeom(const kv_plan *plan, int n_views) {
    const kv_geometry &g = plan->g;
    return RcGeom{g.nx, g.ny, g.nz, g.nu, g.nv, n_views, g.dx, g.dy, g.dz, g.du, g.dv};
}

}  // namespace

kv_status rc_forward_launch(kv_plan *plan, const float *d_src, const float *d_org, int n_views,
                            int mode, const float *vol, const float *meas, float *out, float relax) {
    RcGeom G = rcgeom(plan, n_views);
    dim3 block(32, 4), grid((G.nu + 31) / 32, (G.nv + 3) / 4, n_views);
    cudaStream_t st = plan->ctx->stream;
    LaunchTimer lt(plan->ctx, "rc_fwd");
    switch (mode) {
    case RC_PLAIN: rc_forward_kernel<RC_PLAIN><<<grid, block, 0, st>>>(G, d_src, d_org, vol, meas, out, relax); break;
    case RC_MLEM: rc_forward_kernel<RC_MLEM><<<grid, block, 0, st>>>(G, d_src, d_org, vol, meas, out, relax); break;
    default: rc_forward_kernel<RC_ART><<<grid, block, 0, st>>>(G, d_src, d_org, vol, meas, out, relax); break;
    }
    KV_CHECK_LAUNCH(plan->ctx, "rc_forward_kernel");
    return KV_OK;
}

kv_status rc_build_tables(kv_plan *plan) {
    const RcGeom G = rcgeom(plan, plan->g.n_views);
    const size_t n = (size_t)G.n_views * ((size_t)G.nu + G.nv);
    KV_CHECK_CUDA(plan->ctx, cudaMalloc((void **)&plan->d_rctab, n * sizeof(float)));
    // a block a view: their number has no other limit
    rc_table_kernel<<<G.n_views, 256, 0, plan->ctx->stream>>>(G, plan->d_src, plan->d_org, plan->d_rctab);
    KV_CHECK_LAUNCH(plan->ctx, "rc_table_kernel");
    return KV_OK;
}

kv_status rc_back_slab_launch(kv_plan *plan, int mode, const float *proj, float *vol, int z0, int nzs) {
    if (z0 < 0 || nzs < 1 || z0 + nzs > plan->g.nz)
        return kv_fail(plan->ctx, KV_ERR_INVALID_ARG, "bad slice range for the backprojection");
    RcGeom G = rcgeom(plan, plan->g.n_views);
    dim3 block(32, 4), grid((G.nx + 31) / 32, (G.ny + 4 * kRcRows - 1) / (4 * kRcRows), nzs);
    cudaStream_t st = plan->ctx->stream;
    LaunchTimer lt(plan->ctx, "rc_back");
    switch (mode) {
    case RC_PLAIN: rc_back_kernel<RC_PLAIN><<<grid, block, 0, st>>>(G, plan->d_src, plan->d_org, plan->d_rctab, proj, vol, z0); break;
    case RC_MLEM: rc_back_kernel<RC_MLEM><<<grid, block, 0, st>>>(G, plan->d_src, plan->d_org, plan->d_rctab, proj, vol, z0); break;
    default: rc_back_kernel<RC_ART><<<grid, block, 0, st>>>(G, plan->d_src, plan->d_org, plan->d_rctab, proj, vol, z0); break;
    }
    KV_CHECK_LAUNCH(plan->ctx, "rc_back_kernel");
    return KV_OK;
}

kv_status rc_back_launch(kv_plan *plan, int mode, const float *proj, float *vol) {
    return rc_back_slab_launch(plan, mode, proj, vol, 0, plan->g.nz);
}

kv_status residual_reduce_launch(kv_ctx *ctx, const float *q, const float *p, size_t n, double *red);

kv_status rc_residual_launch(kv_plan *plan, const float *q, const float *p, double *red) {
    return residual_reduce_launch(plan->ctx, q, p, plan->nproj, red);
}

kv_status rc_ratio_launch(kv_plan *plan, int mode, const float *p, float *q, float relax) {
    const int grid = plan->ctx->sm_count > 0 ? plan->ctx->sm_count * 8 : 1024;
    LaunchTimer lt(plan->ctx, "rc_ratio");
    rc_ratio_kernel<<<grid, 256, 0, plan->ctx->stream>>>(mode, p, q, plan->nproj, relax);
    KV_CHECK_LAUNCH(plan->ctx, "rc_ratio_kernel");
    return KV_OK;
}
