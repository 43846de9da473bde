// Index build: pixel selection and compaction, node -> term index, node-pair
// -> term index, symmetric block-row structure and the bin-block CSR layout.
//
// Reference: ImageTermKNNFetcher.cu:19-137, DensityForegroundMapHandler.cu:17-146,
// Node2TermsIndex.cu:8-187, NodePair2TermsIndex.cu:11-296,
// NodePairRowColumnIndex.cu:19-308.
//
// The reference sorts (node, term) and (pair, term) key/value arrays with
// global CUB radix sorts and stable ordering. Both orders are the same as
// sorting unique composite keys (node, term) and (pair, term), so here the
// entries are counted and scattered into per-node segments with integer
// atomics and each short segment is then sorted in shared memory. The result
// is independent of the scatter order, hence bit-exact with the reference
// order and reproducible run to run. No host synchronisation is needed: every
// size lives in DeviceCounts.
#include "kernels_common.cuh"

namespace mvdr {

constexpr uint32_t kChunk = kChunkPixels;

// ----------------------------------------------------- input checks -----
// Node ids of the skinning, the node graph and the correspondences must be
// below num_nodes and surfel ids below num_surfels; otherwise the instance is
// flagged and every kernel that would index with them skips its work.
__global__ void __launch_bounds__(256) input_check_kernel(const InstDesc* insts, uint32_t width, uint32_t height) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
    bool bad = false;
    for (uint32_t i = t0; i < I.S; i += stride) {
        const ushort4 k = I.surfel_knn[i];
        bad |= k.x >= I.N || k.y >= I.N || k.z >= I.N || k.w >= I.N;
    }
    for (uint32_t i = t0; i < I.E; i += stride) {
        const ushort2 e = I.graph[i];
        bad |= e.x >= I.N || e.y >= I.N;
    }
    // selected feature terms take their skinning from the (checked) surfels
    const uint32_t tp = I.feat_select ? 0u : I.Tp;
    for (uint32_t i = t0; i < tp; i += stride) {
        const ushort4 k = I.feat_knn[i];
        bad |= k.x >= I.N || k.y >= I.N || k.z >= I.N || k.w >= I.N;
    }
    for (uint32_t i = t0; i < I.Tc; i += stride) {
        const ushort4 k = I.cross_knn[i];
        bad |= k.x >= I.N || k.y >= I.N || k.z >= I.N || k.w >= I.N;
    }
    const uint32_t npix = width * height;
    for (uint32_t v = 0; v < I.num_views; ++v) {
        const ViewDesc& V = I.views[v];
        for (uint32_t p = t0; p < npix; p += stride) {
            const uint32_t s = V.index[(size_t)(p / width) * V.pitch + p % width];
            bad |= s != kInvalid && s >= I.S;
        }
    }
    if (bad) set_error(I, kErrBadNodeIndex);
}

// ------------------------------------------------------- compaction -----

// a surfel id past the surfel array marks the pixel invalid (and is reported
// by input_check_kernel)
struct DensePred {
    __device__ static inline bool eval(const InstDesc& I, uint32_t v, uint32_t x, uint32_t y) {
        const ViewDesc& V = I.views[v];
        return V.index[(size_t)y * V.pitch + x] < I.S;
    }
};

// markValidColorForegroundMapsPixelKernel (DensityForegroundMapHandler.cu:34-105):
// project the initially warped surfel; keep it when it lands inside the image,
// faces the camera (cos > 0.5) and the filtered mask there is non-zero.
struct ForegroundPred {
    __device__ static inline bool eval(const InstDesc& I, uint32_t v, uint32_t x, uint32_t y) {
        const ViewDesc& V = I.views[v];
        const size_t p = (size_t)y * V.pitch + x;
        const uint32_t s = V.index[p];
        if (!I.use_fg || s >= I.S || V.fg == nullptr || bad_inputs(I)) return false;
        const float4 cv = V.ref_v[p], cn = V.ref_n[p];
        const float3 cv0 = apply3(V.init, mk3(cv.x, cv.y, cv.z));
        const float3 cn0 = rot3(V.init, mk3(cn.x, cn.y, cn.z));
        const M34 se3 = dq_se3(blend_dq(I.se3, I.surfel_knn[s], I.surfel_w[s]));
        const float3 wv = apply3(se3, cv0), wn = rot3(se3, cn0);
        const float3 vc = apply3(V.init_inv, apply3(V.w2c, wv));
        const float3 nc = rot3(V.init_inv, rot3(V.w2c, wn));
        const float inv = rsqrtf(dot3(vc, vc));
        const float cosang = -dot3(mul3(inv, vc), nc);
        const int u = project_coord(vc.x, vc.z, V.fx, V.cx);
        const int w = project_coord(vc.y, vc.z, V.fy, V.cy);
        if (u < 0 || u >= (int)I.width || w < 0 || w >= (int)I.height || !(cosang > 0.5f)) return false;
        return V.fg[(size_t)w * V.pitch + u] > 1e-5f;  // isValidForegroundMaskPixel
    }
};

template <class Pred>
__global__ void __launch_bounds__(256, 6) compact_count_kernel(const InstDesc* insts, uint32_t width, uint32_t height,
                                                            uint32_t cpv) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const uint32_t view = blockIdx.x / cpv, c = blockIdx.x % cpv;
    uint32_t cnt = 0;
    if (view < I.num_views) {
        const uint32_t npix = width * height;
        for (uint32_t k = 0; k < kChunk / 256; ++k) {
            const uint32_t p = c * kChunk + k * 256 + threadIdx.x;
            const bool ok = p < npix && Pred::eval(I, view, p % width, p / width);
            // the write pass reads the predicate back from these bits
            const uint32_t bal = __ballot_sync(0xffffffffu, ok);
            if (lane_id() == 0) I.pix_mask[(size_t)view * cpv * (kChunk / 32) + p / 32] = bal;
            cnt += ok ? 1u : 0u;
        }
    }
    cnt = warp_sum(cnt);
    __shared__ uint32_t ws[8];
    if (lane_id() == 0) ws[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int i = 0; i < 8; ++i) t += ws[i];
        I.chunk_count[blockIdx.x] = t;
    }
}

// exclusive scan of the chunk counts; per-view totals; capacity check
__global__ void __launch_bounds__(1024) compact_scan_kernel(const InstDesc* insts, uint32_t cpv, uint32_t max_views,
                                                            int foreground) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    DeviceCounts* C = I.counts;
    // per-view totals before the scan
    if (threadIdx.x < MVDR_MAX_VIEWS) {
        uint32_t t = 0;
        if (threadIdx.x < max_views)
            for (uint32_t c = 0; c < cpv; ++c) t += I.chunk_count[threadIdx.x * cpv + c];
        if (foreground) C->fg_view_count[threadIdx.x] = t;
        else C->dense_view_count[threadIdx.x] = t;
    }
    __syncthreads();
    uint32_t total = 0;
    __shared__ uint32_t tot;
    block_exclusive_scan_inplace(I.chunk_count, cpv * max_views, &tot);
    __syncthreads();
    if (threadIdx.x == 0) {
        total = tot;
        const uint32_t cap = foreground ? I.cap_fg : I.cap_dense;
        if (total > cap) {
            atomicOr(&C->error_flags, foreground ? kErrForegroundCapacity : kErrDenseCapacity);
            total = cap;
        }
        if (foreground) C->foreground_terms = total;
        else C->dense_terms = total;
    }
}

template <class Pred>
__global__ void __launch_bounds__(256) compact_write_kernel(const InstDesc* insts, uint32_t width, uint32_t height,
                                                            uint32_t cpv, int foreground) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const uint32_t view = blockIdx.x / cpv, c = blockIdx.x % cpv;
    if (view >= I.num_views) return;
    const uint32_t cap = foreground ? I.cap_fg : I.cap_dense;
    __shared__ uint32_t wtot[8];
    uint32_t carry = I.chunk_count[blockIdx.x];
    for (uint32_t k = 0; k < kChunk / 256; ++k) {
        const uint32_t p = c * kChunk + k * 256 + threadIdx.x;
        const uint32_t x = p % width, y = p / width;
        const uint32_t bal = I.pix_mask[(size_t)view * cpv * (kChunk / 32) + p / 32];
        const bool ok = (bal >> lane_id()) & 1u;
        const uint32_t lane_prefix = __popc(bal & ((1u << lane_id()) - 1u));
        if (lane_id() == 0) wtot[threadIdx.x >> 5] = __popc(bal);
        __syncthreads();
        uint32_t wbase = 0, slice = 0;
        for (uint32_t w = 0; w < 8; ++w) {
            if (w < (threadIdx.x >> 5)) wbase += wtot[w];
            slice += wtot[w];
        }
        if (ok) {
            const uint32_t out = carry + wbase + lane_prefix;
            if (out < cap) {
                const ViewDesc& V = I.views[view];
                const uint32_t s = V.index[(size_t)y * V.pitch + x];
                if (s < I.S) {
                    const ushort4 pix = make_ushort4((unsigned short)x, (unsigned short)y, (unsigned short)view, 0);
                    if (foreground) {
                        I.fg_pix[out] = pix;
                        I.fg_knn[out] = I.surfel_knn[s];
                        I.fg_w[out] = I.surfel_w[s];
                    } else {
                        I.dense_pix[out] = pix;
                        I.dense_knn[out] = I.surfel_knn[s];
                        I.dense_w[out] = I.surfel_w[s];
                    }
                } else {
                    set_error(I, kErrBadNodeIndex);
                }
            }
        }
        carry += slice;
        __syncthreads();
    }
}

// view whose maps a compacted pixel samples: its own tag, or in compat mode
// the reference's lookup that reads per-view counts as offsets
// (DenseDepthJacobianResidual.cu:14-22)
__device__ inline uint32_t sample_view(const InstDesc& I, ushort4 pix, uint32_t idx, const uint32_t* view_count) {
    if (!(I.compat & MVDR_COMPAT_REF_VIEW_LOOKUP)) return pix.z;
    for (uint32_t i = 0; i < I.num_views; ++i) {
        if (i == I.num_views - 1) return i;
        if (view_count[i] <= idx && idx < view_count[i + 1]) return i;
    }
    return I.num_views - 1;
}

// canonical vertex / normal of each compacted pixel in frame 0; constant over
// the Gauss-Newton iterations, so computed once per index build
__global__ void __launch_bounds__(256) prepare_pixels_kernel(const InstDesc* insts, bool mixed) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const DeviceCounts* C = I.counts;
    const uint32_t Td = C->dense_terms, Tf = C->foreground_terms;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < Td + Tf; t += gridDim.x * blockDim.x) {
        const bool fg = t >= Td;
        const uint32_t k = fg ? t - Td : t;
        const ushort4 pix = fg ? I.fg_pix[k] : I.dense_pix[k];
        const uint32_t v = sample_view(I, pix, k, fg ? C->fg_view_count : C->dense_view_count);
        const ViewDesc& V = I.views[v];
        const size_t p = (size_t)pix.y * V.pitch + pix.x;
        const float4 cv = V.ref_v[p];
        // the foreground term's vertex stays in its camera's frame in the
        // reference's form (density_map_jacobian.cuh:32-36)
        const bool raw_frame = fg && (I.compat & MVDR_COMPAT_REF_FOREGROUND_FRAME);
        float3 a = raw_frame ? mk3(cv.x, cv.y, cv.z) : apply3(V.init, mk3(cv.x, cv.y, cv.z));
        if (!fg && mixed) {
            // The point-to-plane residual subtracts two ~1 m positions, and
            // near convergence Jt r cancels by orders of magnitude more, so
            // the FP32 rounding of this transform (~1e-7 m) would dominate
            // the increment. Keep the transform in double as hi + lo floats.
            const double* m = V.init_d;
            double ad[3];
#pragma unroll
            for (int r = 0; r < 3; ++r)
                ad[r] = m[3 * r] * (double)cv.x + m[3 * r + 1] * (double)cv.y + m[3 * r + 2] * (double)cv.z + m[9 + r];
            a = mk3((float)ad[0], (float)ad[1], (float)ad[2]);
            I.dense_cv_lo[k] = make_float4((float)(ad[0] - (double)a.x), (float)(ad[1] - (double)a.y),
                                           (float)(ad[2] - (double)a.z), 0.f);
        }
        if (fg) {
            I.fg_cv[k] = make_float4(a.x, a.y, a.z, __uint_as_float(v));
        } else {
            const float4 cn = V.ref_n[p];
            const float3 b = rot3(V.init, mk3(cn.x, cn.y, cn.z));
            // the rendered grey level of the density term: rgb2density of the
            // normalised rgb solver map (ColorTypeTransfer.h:51-56,
            // DensityForegroundJacobianResidual.cu:51-52)
            float geo = 0.f;
            if (I.use_density) {
                const float4 c = V.rgb[p];
                geo = 0.299f * c.x + 0.587f * c.y + 0.114f * c.z;
            }
            I.dense_cv[k] = make_float4(a.x, a.y, a.z, __uint_as_float(v));
            I.dense_cn[k] = make_float4(b.x, b.y, b.z, geo);
        }
    }
}

// ------------------------------------------- sparse feature selection -----
// SparseCorrespondenceHandler (SparseCorrespondenceHandler.cu:18-199), the
// nearest-distance form (USE_NEAREST_DISTANCE_PAIRS, solver_constants.h:9).
// Maps are read with the reference's border addressing: outside the image a
// float4 map reads zero and the index map reads 0, which counts as a surfel
// (it is not 0xFFFFFFFF); such a pixel's coordinate then wraps to 0xFFFF as
// an unsigned short and fails the image-size test, as in the reference.

__device__ inline float4 border4(const float4* m, int x, int y, uint32_t W, uint32_t H, uint32_t pitch) {
    if (x < 0 || y < 0 || x >= (int)W || y >= (int)H) return make_float4(0.f, 0.f, 0.f, 0.f);
    return m[(size_t)y * pitch + x];
}

// is_zero_vertex (VectorUtils.h:214-216): the 1e-3 bound is a double
__device__ inline bool zero_vertex4(float4 v) {
    return (double)fabsf(v.x) < 1e-3 && (double)fabsf(v.y) < 1e-3 && (double)fabsf(v.z) < 1e-3;
}

// The selection's float arithmetic is written with round-to-nearest
// intrinsics, which the compiler does not contract into FMAs: the kept pairs
// and the term positions are then the CPU restatement's to the bit (a one-ulp
// shift of a target moves the small late-iteration residuals measurably).
__device__ inline float sq_dist3(float4 a, float4 b) {
    const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// m * p + t, uncontracted (mat34 applied as the reference writes it)
__device__ inline float3 apply3_rn(const M34& m, float3 p) {
    float o[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        o[r] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m.r[3 * r], p.x), __fmul_rn(m.r[3 * r + 1], p.y)),
                                   __fmul_rn(m.r[3 * r + 2], p.z)),
                         m.t[r]);
    return mk3(o[0], o[1], o[2]);
}

// chooseValidPixelKernel: one thread per candidate pair
__global__ void __launch_bounds__(256) feat_choose_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    if (!I.feat_select) return;
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= I.fp_offset[MVDR_MAX_VIEWS]) return;
    uint32_t v = 0;
    while (v + 1 < I.num_views && idx >= I.fp_offset[v + 1]) ++v;
    const ViewDesc& V = I.views[v];
    const uint32_t W = I.width, H = I.height, P = V.pitch;
    const ushort4 pair = I.fp_pairs[v][idx - I.fp_offset[v]];
    // validDepthPixelInWindow: the last row's first non-zero vertex, the
    // centre preferred
    ushort2 dp = make_ushort2(0xFFFF, 0xFFFF);
    for (int y = (int)pair.w - 1; y <= (int)pair.w + 1; ++y)
        for (int x = (int)pair.z - 1; x <= (int)pair.z + 1; ++x)
            if (!zero_vertex4(border4(V.obs_v, x, y, W, H, P))) {
                dp = make_ushort2((unsigned short)x, (unsigned short)y);
                break;
            }
    if (!zero_vertex4(border4(V.obs_v, pair.z, pair.w, W, H, P))) dp = make_ushort2(pair.z, pair.w);
    uint32_t keep = 0;
    ushort4 chosen = make_ushort4(0, 0, 0, 0);
    const uint8_t* edge = I.fp_edge[v];
    const bool on_edge = edge && dp.x < W && dp.y < H && edge[(size_t)dp.y * P + dp.x] == 1;
    if (dp.x < W && dp.y < H && !on_edge) {
        const float4 ov = V.obs_v[(size_t)dp.y * P + dp.x];
        // validGeometryPixelInWindow (nearest form): the window pixel with a
        // surfel whose live vertex is nearest the observed vertex
        ushort2 gp = make_ushort2(0xFFFF, 0xFFFF);
        float best = 100.0f;
        for (int y = (int)pair.y - 1; y <= (int)pair.y + 1; ++y)
            for (int x = (int)pair.x - 1; x <= (int)pair.x + 1; ++x) {
                const bool in = x >= 0 && y >= 0 && x < (int)W && y < (int)H;
                const uint32_t s = in ? V.index[(size_t)y * P + x] : 0u;
                if (s != kInvalid) {
                    const float d = sq_dist3(ov, border4(I.fp_live[v], x, y, W, H, P));
                    if (d < best) {
                        gp = make_ushort2((unsigned short)x, (unsigned short)y);
                        best = d;
                    }
                }
            }
        if (gp.x < W && gp.y < H) {
            const size_t o = (size_t)gp.y * P + gp.x;
            const uint32_t s = V.index[o];
            // a pixel without a valid surfel id cannot give a skinning
            if (s < I.S && sq_dist3(V.ref_v[o], ov) < 2.5e-3f) {
                keep = 1;
                chosen = make_ushort4(gp.x, gp.y, dp.x, dp.y);
            }
        }
    }
    I.fp_keep[idx] = keep;
    I.fp_chosen[idx] = chosen;
}

// compactQueryValidPairsKernel: kept pairs in candidate order (one CTA of
// 1024 threads per instance: an exclusive scan of the keep flags, then each
// kept pair written at its prefix)
__global__ void __launch_bounds__(1024) feat_compact_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    if (!I.feat_select) return;
    const uint32_t n = I.fp_offset[MVDR_MAX_VIEWS];
    __shared__ uint32_t total;
    block_exclusive_scan_inplace(I.fp_keep, n, &total);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t o = I.fp_keep[i];
        const uint32_t next = i + 1 < n ? I.fp_keep[i + 1] : total;
        if (next == o) continue;
        uint32_t v = 0;
        while (v + 1 < I.num_views && i >= I.fp_offset[v + 1]) ++v;
        const ViewDesc& V = I.views[v];
        const ushort4 c = I.fp_chosen[i];
        const size_t og = (size_t)c.y * V.pitch + c.x, oo = (size_t)c.w * V.pitch + c.z;
        const float4 rv = V.ref_v[og];
        const float3 r0 = apply3_rn(V.init, mk3(rv.x, rv.y, rv.z));
        const float4 dv = V.obs_v[oo];
        const float3 t0 = apply3_rn(V.c2w, apply3_rn(V.init, mk3(dv.x, dv.y, dv.z)));
        const uint32_t s = V.index[og];
        I.fp_target[o] = make_float4(t0.x, t0.y, t0.z, 1.0f);
        I.fp_ref[o] = make_float4(r0.x, r0.y, r0.z, rv.w);
        I.fp_knn[o] = I.surfel_knn[s];
        I.fp_w[o] = I.surfel_w[s];
    }
    if (threadIdx.x == 0) I.counts->feature_terms = total;
}

// size2offset (term_offset_types.h:44-64) on the device
__global__ void term_offsets_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    if (threadIdx.x != 0) return;
    DeviceCounts* C = I.counts;
    C->smooth_terms = I.E;
    // selected feature terms: their count was written by feat_compact_kernel
    const uint32_t tp = I.feat_select ? C->feature_terms : I.Tp;
    C->feature_terms = tp;
    C->cross_terms = I.Tc;
    uint32_t o = C->dense_terms;
    C->term_offset[0] = o;
    o += I.E;
    C->term_offset[1] = o;
    o += C->foreground_terms;
    C->term_offset[2] = o;
    o += tp;
    C->term_offset[3] = o;
    o += I.Tc;
    C->term_offset[4] = o;
}

// ------------------------------------------------------ node -> term -----

// Neighbouring pixels share their KNN nodes, so the lanes of a warp that
// hold the same node are merged (match_any) and one lane adds the group's
// count: one atomic per distinct node and slot in the warp.
__global__ void __launch_bounds__(256) n2t_count_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    if (bad_inputs(I)) return;
    TermOffsets off;
    off.load(I.counts);
    const uint32_t T = off.o[4], lane = lane_id();
    const uint32_t stride = gridDim.x * blockDim.x;
    // the warp's 32 terms per step, so that every lane takes part in the match
    for (uint32_t tw = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); tw < T; tw += stride) {
        const uint32_t t = tw + lane;
        uint32_t a[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
        if (t < T) {
            uint32_t k;
            const TermType ty = off.typed(t, k);
            const ushort4 n = term_nodes(I, ty, k);
            const uint32_t m = ty == kSmooth ? 2 : 4;
            const unsigned short v[4] = {n.x, n.y, n.z, n.w};
            for (uint32_t j = 0; j < m; ++j) {
                if (v[j] < I.N) a[j] = v[j];
                else set_error(I, kErrBadNodeIndex);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t grp = __match_any_sync(0xffffffffu, a[j]);
            if (a[j] != 0xFFFFFFFFu && lane == (uint32_t)(__ffs(grp) - 1))
                atomicAdd(&I.n2t_count[a[j]], (uint32_t)__popc(grp));
        }
    }
}
// single-CTA exclusive scans over per-node arrays
enum ScanWhat : int { kScanN2T = 0, kScanRows = 1, kScanUpper = 2, kScanBlkRows = 3, kScanBins = 4 };

__global__ void __launch_bounds__(1024) node_scan_kernel(const InstDesc* insts, int what) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    DeviceCounts* C = I.counts;
    __shared__ uint32_t total;
    const uint32_t N = I.N;
    switch (what) {
        case kScanN2T: {
            for (uint32_t i = threadIdx.x; i <= N; i += blockDim.x) {
                I.n2t_offset[i] = i < N ? I.n2t_count[i] : 0u;
                if (i < N) I.n2t_cursor[i] = 0;
            }
            __syncthreads();
            block_exclusive_scan_inplace(I.n2t_offset, N + 1, &total);
            __syncthreads();
            if (threadIdx.x == 0) {
                C->node2term_entries = total;
                if (total > I.cap_k1) atomicOr(&C->error_flags, kErrNode2TermCapacity);
            }
            break;
        }
        case kScanRows: {
            for (uint32_t i = threadIdx.x; i <= N; i += blockDim.x) I.row_offset[i] = i < N ? I.row_count[i] : 0u;
            __syncthreads();
            block_exclusive_scan_inplace(I.row_offset, N + 1, &total);
            __syncthreads();
            if (threadIdx.x == 0) {
                C->nodepair_entries = total;
                if (total > I.cap_k2) atomicOr(&C->error_flags, kErrNodePairEntryCapacity);
            }
            break;
        }
        case kScanUpper: {
            for (uint32_t i = threadIdx.x; i <= N; i += blockDim.x) {
                I.half_offset[i] = i < N ? I.upper_count[i] : 0u;
                if (i < N) { I.lower_count[i] = 0; I.lower_cursor[i] = 0; }
            }
            __syncthreads();
            block_exclusive_scan_inplace(I.half_offset, N + 1, &total);
            __syncthreads();
            if (threadIdx.x == 0) {
                C->half_pairs = total;
                if (total > I.cap_pairs) atomicOr(&C->error_flags, kErrHalfPairCapacity);
            }
            break;
        }
        case kScanBlkRows: {
            for (uint32_t i = threadIdx.x; i <= N; i += blockDim.x)
                I.blkrow_offset[i] = i < N ? I.lower_count[i] + I.upper_count[i] : 0u;
            __syncthreads();
            block_exclusive_scan_inplace(I.blkrow_offset, N + 1, &total);
            break;
        }
        case kScanBins: {
            const uint32_t nb = C->num_bins;
            __syncthreads();
            block_exclusive_scan_inplace(I.bin_scan, nb + 1, &total);
            __syncthreads();
            if (threadIdx.x == 0) {
                C->binblock_nnz = I.bin_scan[nb];
                if (I.bin_scan[nb] > I.cap_bb) atomicOr(&C->error_flags, kErrBinBlockCapacity);
            }
            break;
        }
        default: break;
    }
}

// The same grouping: the group's first lane reserves the group's slots and
// every lane takes its rank in the group (the sort that follows orders them).
__global__ void __launch_bounds__(256) n2t_scatter_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    TermOffsets off;
    off.load(I.counts);
    const uint32_t T = off.o[4], lane = lane_id();
    const uint32_t K1 = I.counts->node2term_entries;
    if (K1 > I.cap_k1) return;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t tw = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); tw < T; tw += stride) {
        const uint32_t t = tw + lane;
        uint32_t a[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
        if (t < T) {
            uint32_t k;
            const TermType ty = off.typed(t, k);
            const ushort4 n = term_nodes(I, ty, k);
            const uint32_t m = ty == kSmooth ? 2 : 4;
            const unsigned short v[4] = {n.x, n.y, n.z, n.w};
            for (uint32_t j = 0; j < m; ++j)
                if (v[j] < I.N) a[j] = v[j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t grp = __match_any_sync(0xffffffffu, a[j]);
            const uint32_t leader = __ffs(grp) - 1;
            uint32_t base = 0;
            if (a[j] != 0xFFFFFFFFu && lane == leader) base = atomicAdd(&I.n2t_cursor[a[j]], (uint32_t)__popc(grp));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (a[j] != 0xFFFFFFFFu)
                I.n2t_index[I.n2t_offset[a[j]] + base + __popc(grp & ((1u << lane) - 1u))] = t;
        }
    }
}

// Ascending sort of 32 kSlots keys in a warp's registers: element
// i = 32 s + lane sits in slot s of a lane; a bitonic network exchanges across
// lanes with shuffles (partner distance < 32) and inside a lane between slots
// otherwise.
template <int kSlots> __device__ inline void warp_sort(uint32_t (&v)[kSlots]) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (uint32_t k = 2; k <= 32u * kSlots; k <<= 1) {
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                const int sj = (int)(j >> 5);
#pragma unroll
                for (int sl = 0; sl < kSlots; ++sl) {
                    if (sl & sj) continue;
                    const uint32_t i = 32u * sl + lane;
                    const bool up = (i & k) == 0;
                    const uint32_t a = v[sl], c = v[sl | sj];
                    v[sl] = up ? min(a, c) : max(a, c);
                    v[sl | sj] = up ? max(a, c) : min(a, c);
                }
            } else {
#pragma unroll
                for (int sl = 0; sl < kSlots; ++sl) {
                    const uint32_t i = 32u * sl + lane;
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, v[sl], j);
                    const bool up = (i & k) == 0, lower = (i & j) == 0;
                    v[sl] = (up == lower) ? min(v[sl], o) : max(v[sl], o);
                }
            }
        }
    }
}

// Each node's term segment ascending. Up to kSortRun terms: a warp per node.
constexpr int kSortSlots = 8;
constexpr uint32_t kSortRun = 32u * kSortSlots, kMergeMax = 4096;

__global__ void __launch_bounds__(256) n2t_warp_sort_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    if (I.counts->node2term_entries > I.cap_k1) return;
    const uint32_t lane = lane_id();
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t node = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); node < I.N; node += warps) {
        const uint32_t b = I.n2t_offset[node], e = I.n2t_offset[node + 1];
        const uint32_t len = e - b;
        if (len <= 1 || len > kSortRun) continue;
        if (len > I.cap_seg) {  // the segment exceeds max_terms_per_node
            if (lane == 0) set_error(I, kErrSegmentTooLong);
            continue;
        }
        uint32_t v[kSortSlots];
#pragma unroll
        for (int sl = 0; sl < kSortSlots; ++sl) {
            const uint32_t i = 32u * sl + lane;
            v[sl] = i < len ? I.n2t_index[b + i] : 0xFFFFFFFFu;
        }
        warp_sort<kSortSlots>(v);
#pragma unroll
        for (int sl = 0; sl < kSortSlots; ++sl) {
            const uint32_t i = 32u * sl + lane;
            if (i < len) I.n2t_index[b + i] = v[sl];
        }
    }
}

// From kSortRun to kMergeMax terms: a CTA per node. Its warps sort runs of
// kSortRun in registers; each key's place is then its place in its run plus the
// number of smaller keys in every other run (binary searches in shared memory).
// A warp with 16 or 32 slots, or a bitonic sort over shared memory, has a chain of
// 45 to 78 exchange steps per node: 106 -> 21 us on a 500-node frame, 413 -> 257
// us on 32,768 nodes.
constexpr uint32_t kMergeWarps = 4;

__global__ void __launch_bounds__(32 * kMergeWarps) n2t_merge_sort_kernel(const InstDesc* insts) {
    chain_wait();
    __shared__ uint32_t key[kMergeMax];
    const InstDesc& I = insts[blockIdx.y];
    if (I.counts->node2term_entries > I.cap_k1) return;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    for (uint32_t node = blockIdx.x; node < I.N; node += gridDim.x) {
        const uint32_t b = I.n2t_offset[node], len = I.n2t_offset[node + 1] - b;
        if (len <= kSortRun) continue;
        if (len > I.cap_seg) {
            if (threadIdx.x == 0) set_error(I, kErrSegmentTooLong);
            continue;
        }
        if (len > kMergeMax) continue;  // n2t_sort_kernel's
        const uint32_t runs = (len + kSortRun - 1) / kSortRun;
        for (uint32_t r = warp; r < runs; r += kMergeWarps) {
            uint32_t v[kSortSlots];
#pragma unroll
            for (int sl = 0; sl < kSortSlots; ++sl) {
                const uint32_t i = kSortRun * r + 32u * sl + lane;
                v[sl] = i < len ? I.n2t_index[b + i] : 0xFFFFFFFFu;
            }
            warp_sort<kSortSlots>(v);
#pragma unroll
            for (int sl = 0; sl < kSortSlots; ++sl) key[kSortRun * r + 32u * sl + lane] = v[sl];
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < len; i += 32 * kMergeWarps) {
            // (only the last run is padded, with keys above every term)
            const uint32_t r = i / kSortRun, k = key[i];
            uint32_t rank = i % kSortRun;
            for (uint32_t o = 0; o < runs; ++o) {
                if (o == r) continue;
                // keys below k, and for an earlier run also those equal to it
                const uint32_t* run = key + kSortRun * o;
                uint32_t n = 0;
#pragma unroll
                for (uint32_t step = kSortRun / 2; step > 0; step >>= 1) {
                    const uint32_t x = run[n + step - 1];
                    if (x < k || (o < r && x == k)) n += step;
                }
                const uint32_t x = run[n];
                if (x < k || (o < r && x == k)) ++n;
                rank += n;
            }
            I.n2t_index[b + rank] = k;
        }
        __syncthreads();
    }
}

// longer segments: a bitonic sort in shared memory, one CTA per node
__global__ void __launch_bounds__(256) n2t_sort_kernel(const InstDesc* insts) {
    chain_wait();
    extern __shared__ uint32_t s32[];
    const InstDesc& I = insts[blockIdx.y];
    if (I.counts->node2term_entries > I.cap_k1) return;
    for (uint32_t node = blockIdx.x; node < I.N; node += gridDim.x) {
        const uint32_t b = I.n2t_offset[node], e = I.n2t_offset[node + 1];
        const uint32_t len = e - b;
        if (len <= kMergeMax || len > I.cap_seg) continue;
        const uint32_t n2 = next_pow2(len);
        for (uint32_t i = threadIdx.x; i < n2; i += blockDim.x) s32[i] = i < len ? I.n2t_index[b + i] : 0xFFFFFFFFu;
        __syncthreads();
        block_bitonic_sort(s32, n2);
        for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) I.n2t_index[b + i] = s32[i];
        __syncthreads();
    }
}

// ------------------------------------------------ node pair -> term -----
// Row i of the upper triangle holds the entries (j, t) for every term t of
// node i and every other node j > i of t: the reference's half-pair keys
// (computeKVNodePairKNN, NodePair2TermsIndex.cu:11-28; smooth pairs :71-81)
// grouped by their smaller node.

__device__ inline uint32_t upper_entries_of(const InstDesc& I, const TermOffsets& off, uint32_t node, uint32_t t,
                                            uint32_t js[4]) {
    uint32_t k;
    const TermType ty = off.typed(t, k);
    const ushort4 n = term_nodes(I, ty, k);
    uint32_t c = 0;
    if (ty == kSmooth) {
        // the smooth term contributes one pair (min, max) to the row of min
        const uint32_t a = n.x, b = n.y;
        if (a == node && b > node && b < I.N) js[c++] = b;
        else if (b == node && a > node && a < I.N) js[c++] = a;
        // a node listed twice in the same smooth term (a == b) gives no pair
        return c;
    }
    const unsigned short a[4] = {n.x, n.y, n.z, n.w};
    for (int q = 0; q < 4; ++q)
        if (a[q] > node && a[q] < I.N) js[c++] = a[q];
    return c;
}

constexpr uint32_t kRowWarps = 4;  // of a CTA of the two row kernels

// W warps (1, or the CTA's) per node: number of upper entries of the row, and n2t_w[p], the node's
// skinning weight in each of its terms (0 for smooth; the values are those of
// weight_of, PreconditionerBlocked.cu:23-29). The weights are inputs, recorded
// once per solve, so that the assembly kernels read one coalesced value per entry
// instead of the term's node and weight records.
template <uint32_t W>
__global__ void __launch_bounds__(32 * kRowWarps) np_row_count_kernel(const InstDesc* insts) {
    chain_wait();
    __shared__ uint32_t s_sum[kRowWarps];
    const InstDesc& I = insts[blockIdx.y];
    if (I.counts->node2term_entries > I.cap_k1) return;
    TermOffsets off;
    off.load(I.counts);
    constexpr uint32_t kNodes = kRowWarps / W;
    const uint32_t warp = threadIdx.x >> 5, sub = warp % W;
    for (uint32_t n0 = blockIdx.x * kNodes; n0 < I.N; n0 += gridDim.x * kNodes) {
        const uint32_t node = n0 + warp / W;
        uint32_t c = 0;
        if (node < I.N) {
            const uint32_t b = I.n2t_offset[node], e = I.n2t_offset[node + 1];
#pragma unroll 4
            for (uint32_t p = b + 32 * sub + lane_id(); p < e; p += 32 * W) {
                uint32_t k;
                const TermType ty = off.typed(I.n2t_index[p], k);
                const ushort4 n = term_nodes(I, ty, k);
                float w = 0.f;
                if (ty == kSmooth) {
                    // one pair (min, max), in the row of min; a node listed twice in
                    // the same smooth term gives no pair
                    const uint32_t o = n.x == node ? n.y : n.x;
                    c += o > node && o < I.N ? 1u : 0u;
                } else {
                    if (ty != kInvalidTerm) w = weight_of(n, term_weights(I, ty, k), node);
                    const uint32_t a[4] = {n.x, n.y, n.z, n.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) c += a[q] > node && a[q] < I.N ? 1u : 0u;
                }
                I.n2t_w[p] = w;
            }
            c = warp_sum(c);
            if (W == 1 && lane_id() == 0) I.row_count[node] = c;
        }
        if constexpr (W > 1) {
            if (lane_id() == 0) s_sum[warp] = c;
            __syncthreads();
            if (sub == 0 && lane_id() == 0 && node < I.N) {
                for (uint32_t w = 1; w < W; ++w) c += s_sum[warp + w];
                I.row_count[node] = c;
            }
            __syncthreads();
        }
    }
}

// W warps per node: the row's (j, t) entries, j > node, in ascending (j, t) order
// without sorting, with the products of the two nodes' weights. The node's term
// list is already ascending in t. A first pass counts the entries of each
// distinct partner in a small hash table in shared memory; the partners are
// ranked, which gives each one's start; a second pass places the entries: of 32
// consecutive terms, those of the same partner take consecutive places in lane
// order. Both passes take kRowSlices slices of 32 terms at once, so that their
// gathers overlap; bound by those gathers and by the table's traffic in shared memory
// (32,768 nodes: that pipe 58 % busy, a third of the warps): with four slices (80
// registers) 32,768 nodes take 929 us and 500 nodes the same 101, with one 580 and 118. A term that lists a partner twice, or a
// node with more than kRowPartners partners, takes the sweep (one pass over the
// list per partner), which is what every node took before: 285 -> 101 us on a
// 500-node frame, whose lists reach 1,276 terms (54 with a CTA per node), 72 -> 51 us
// on 4,096 nodes, 752 -> 606 us on 32,768, with the weights' own pass (77, 42 and 219
// us) saved. Writes np_index, np_scale, the per-pair (key, start) of the row and
// upper_count.
constexpr uint32_t kRowSlices = 2, kRowPartners = 192;

// W warps of a CTA share the table and a node's list, a run of it each
template <uint32_t W> struct RowTable {
    static constexpr uint32_t kBits = W == 1 ? 8 : 9, kSize = 1u << kBits;
    // every thread may pass the test of `used` before the others' insertions count
    static_assert(kRowPartners + 32 * W < kSize, "a free entry must remain");
    uint32_t key[kSize];       // partner, kInvalid: free
    uint32_t count[W][kSize];  // its entries in the warp's run, then the place of the next one
    uint32_t mask[W][kSize];   // lanes of the warp's current slice that hold it
    uint32_t slot[kRowPartners], rank_slot[kRowPartners];  // the used slots, then in order of the partner
    uint32_t used, sweep;

    __device__ static uint32_t hash(uint32_t j) { return (j * 2654435761u) >> (32 - kBits); }
    __device__ static uint32_t next(uint32_t h) { return (h + 1) & (kSize - 1); }
    __device__ uint32_t find(uint32_t j) const {
        uint32_t h = hash(j);
        while (key[h] != j) h = next(h);
        return h;
    }
};

// weight product of an entry's two nodes, exact in double (0 for a smooth term)
__device__ inline double pair_scale(const InstDesc& I, const TermOffsets& off, uint32_t t, uint32_t i, uint32_t j) {
    uint32_t k;
    const TermType ty = off.typed(t, k);
    if (ty == kSmooth || ty == kInvalidTerm) return 0.0;
    const ushort4 kn = term_nodes(I, ty, k);
    const float4 w4 = term_weights(I, ty, k);
    return (double)weight_of(kn, w4, i) * (double)weight_of(kn, w4, j);
}

// the sweep: for each distinct partner (ascending, found by a warp minimum) one
// pass over the list emits the terms that contain it, in t order, and finds the
// next partner. A term that lists a partner twice contributes two adjacent
// entries, like the duplicate keys of a sort. Returns the distinct partners.
__device__ inline uint32_t row_sweep(const InstDesc& I, const TermOffsets& off, uint32_t node, uint32_t b0, uint32_t b1,
                                     uint32_t out, uint32_t len) {
    const uint32_t lane = lane_id();
    uint32_t pos = 0, runs = 0, j = node;  // the first pass emits nothing and finds the first partner
    for (bool first = true;; first = false) {
        if (!first && lane == 0 && pos < len) {
            I.tmp_key[out + runs] = node * I.enc + j;
            I.tmp_start[out + runs] = out + pos;
        }
        uint32_t nxt = 0xFFFFFFFFu;
        for (uint32_t base = b0; base < b1; base += 32) {
            const uint32_t p = base + lane, t = p < b1 ? I.n2t_index[p] : kInvalid;
            uint32_t js[4], mult = 0;
            const uint32_t c = p < b1 ? upper_entries_of(I, off, node, t, js) : 0u;
            for (uint32_t q = 0; q < c; ++q) {
                if (!first && js[q] == j) ++mult;
                if (js[q] > j) nxt = min(nxt, js[q]);
            }
            const uint32_t incl = warp_inclusive_scan(mult), total = __shfl_sync(0xffffffffu, incl, 31);
            for (uint32_t m = 0; m < mult; ++m) {
                const uint32_t at = pos + incl - mult + m;
                if (at >= len) break;
                I.np_index[out + at] = t;
                I.np_scale[out + at] = pair_scale(I, off, t, node, j);
            }
            pos += total;
        }
        if (!first) ++runs;
        j = warp_min_u32(nxt);
        if (j == 0xFFFFFFFFu) return runs;
    }
}

template <uint32_t W>
__global__ void __launch_bounds__(32 * kRowWarps, 8) np_row_build_kernel(const InstDesc* insts) {
    chain_wait();
    static_assert(W == 1 || W == kRowWarps, "a warp or the CTA");
    using Table = RowTable<W>;
    __shared__ Table s_table[kRowWarps / W];
    const InstDesc& I = insts[blockIdx.y];
    const DeviceCounts* C = I.counts;
    if (C->node2term_entries > I.cap_k1 || C->nodepair_entries > I.cap_k2) return;
    TermOffsets off;
    off.load(I.counts);
    const uint32_t lane = lane_id(), lt_mask = (1u << lane) - 1u;
    const uint32_t warp = threadIdx.x >> 5, sub = warp % W, member = 32 * sub + lane;
    Table& tb = s_table[warp / W];
    uint32_t* const count = tb.count[sub];
    uint32_t* const mask = tb.mask[sub];
    auto sync = [] {
        if constexpr (W == 1) __syncwarp();
        else __syncthreads();
    };
    constexpr uint32_t kNodes = kRowWarps / W;  // (W > 1: the same node for every thread)
    for (uint32_t node = blockIdx.x * kNodes + warp / W; node < I.N; node += gridDim.x * kNodes) {
        const uint32_t b0 = I.n2t_offset[node], b1 = I.n2t_offset[node + 1];
        const uint32_t out = I.row_offset[node], len = I.row_count[node];
        // this warp's run of the list
        const uint32_t run = (b1 - b0 + 32 * W - 1) / (32 * W) * 32;
        const uint32_t c0 = min(b0 + sub * run, b1), c1 = min(c0 + run, b1);
        for (uint32_t i = member; i < Table::kSize; i += 32 * W) {
            tb.key[i] = kInvalid;
#pragma unroll
            for (uint32_t w = 0; w < W; ++w) tb.count[w][i] = tb.mask[w][i] = 0;
        }
        if (member == 0) tb.used = tb.sweep = 0;
        sync();
        // the partners above `node` of the terms of kRowSlices slices
        uint32_t t[kRowSlices], js[kRowSlices][4];
        auto load = [&](uint32_t base) {
#pragma unroll
            for (uint32_t s = 0; s < kRowSlices; ++s) {
                const uint32_t p = base + 32 * s + lane;
                t[s] = p < c1 ? I.n2t_index[p] : kInvalid;
            }
#pragma unroll
            for (uint32_t s = 0; s < kRowSlices; ++s) {
                uint32_t k;
                const TermType ty = off.typed(t[s], k);
                const ushort4 n = t[s] != kInvalid ? term_nodes(I, ty, k) : make_ushort4(0xFFFF, 0xFFFF, 0xFFFF, 0xFFFF);
                const uint32_t a[4] = {n.x, n.y, n.z, n.w};
                if (ty == kSmooth) {  // one pair (min, max), in the row of min
                    const uint32_t o = a[0] == node ? a[1] : a[0];
                    js[s][0] = o > node && o < I.N ? o : kInvalid;
                    js[s][1] = js[s][2] = js[s][3] = kInvalid;
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) js[s][q] = a[q] > node && a[q] < I.N ? a[q] : kInvalid;
                }
            }
        };
        bool sweep = false;
        for (uint32_t base = c0; base < c1 && !sweep; base += 32 * kRowSlices) {
            load(base);
#pragma unroll
            for (uint32_t s = 0; s < kRowSlices; ++s) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t j = js[s][q];
                    if (j == kInvalid) continue;
                    bool twice = false;
#pragma unroll
                    for (int o = 0; o < q; ++o) twice |= js[s][o] == j;
                    if (twice || *(volatile uint32_t*)&tb.used >= kRowPartners) {
                        tb.sweep = 1;
                        continue;
                    }
                    uint32_t h = Table::hash(j);
                    for (;;) {
                        const uint32_t seen = atomicCAS(&tb.key[h], kInvalid, j);
                        if (seen == j) break;
                        if (seen == kInvalid) {
                            const uint32_t u = atomicAdd(&tb.used, 1u);
                            if (u < kRowPartners) tb.slot[u] = h;
                            break;
                        }
                        h = Table::next(h);
                    }
                    atomicAdd(&count[h], 1u);
                }
            }
            __syncwarp();
            sweep = __any_sync(0xffffffffu, *(volatile uint32_t*)&tb.sweep != 0);  // (the same in every lane)
        }
        sync();
        const uint32_t used = tb.used;
        if (tb.sweep || used > kRowPartners) {
            if (sub == 0) {
                const uint32_t runs = row_sweep(I, off, node, b0, b1, out, len);
                if (lane == 0) I.upper_count[node] = runs;
            }
            sync();
            continue;
        }
        // rank the partners; starts in that order, within a partner in order of the runs
        for (uint32_t i = member; i < used; i += 32 * W) {
            const uint32_t h = tb.slot[i], j = tb.key[h];
            uint32_t rank = 0;
            for (uint32_t m = 0; m < used; ++m) rank += tb.key[tb.slot[m]] < j ? 1u : 0u;
            tb.rank_slot[rank] = h;
        }
        sync();
        if (sub == 0) {
            uint32_t start = 0;
            for (uint32_t base = 0; base < used; base += 32) {
                const uint32_t r = base + lane, h = r < used ? tb.rank_slot[r] : 0u;
                uint32_t n = 0;
                for (uint32_t w = 0; w < W; ++w) n += r < used ? tb.count[w][h] : 0u;
                const uint32_t incl = warp_inclusive_scan(n);
                uint32_t place = start + incl - n;
                if (r < used) {
                    I.tmp_key[out + r] = node * I.enc + tb.key[h];
                    I.tmp_start[out + r] = out + place;
                    for (uint32_t w = 0; w < W; ++w) {
                        const uint32_t own = tb.count[w][h];
                        tb.count[w][h] = place;
                        place += own;
                    }
                }
                start += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) I.upper_count[node] = used;
        }
        sync();
        // place the entries
        for (uint32_t base = c0; base < c1; base += 32 * kRowSlices) {
            load(base);
            float4 w4[kRowSlices];
            ushort4 kn[kRowSlices];
#pragma unroll
            for (uint32_t s = 0; s < kRowSlices; ++s) {
                uint32_t k;
                const TermType ty = off.typed(t[s], k);
                const bool weighted = t[s] != kInvalid && ty != kSmooth && ty != kInvalidTerm;
                kn[s] = weighted ? term_nodes(I, ty, k) : make_ushort4(0, 0, 0, 0);
                w4[s] = weighted ? term_weights(I, ty, k) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (uint32_t s = 0; s < kRowSlices; ++s) {
                uint32_t h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    h[q] = kInvalid;
                    if (js[s][q] == kInvalid) continue;
                    h[q] = tb.find(js[s][q]);
                    atomicOr(&mask[h[q]], 1u << lane);
                }
                __syncwarp();
                const double wi = (double)weight_of(kn[s], w4[s], node);
                uint32_t m[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (h[q] == kInvalid) continue;
                    m[q] = mask[h[q]];
                    const uint32_t at = count[h[q]] + __popc(m[q] & lt_mask);
                    if (at < len) {
                        I.np_index[out + at] = t[s];
                        I.np_scale[out + at] = wi * (double)weight_of(kn[s], w4[s], js[s][q]);
                    }
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 4; ++q) {  // the partner's first lane moves its place on
                    if (h[q] == kInvalid || (m[q] & lt_mask)) continue;
                    count[h[q]] += __popc(m[q]);
                    mask[h[q]] = 0;
                }
                __syncwarp();
            }
        }
        sync();
    }
}

// warp per node: copy the row's unique pairs to the compact half-pair arrays
// and count the lower-triangle entries of each column
__global__ void __launch_bounds__(256) np_half_compact_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const DeviceCounts* C = I.counts;
    if (C->half_pairs > I.cap_pairs || C->nodepair_entries > I.cap_k2 || C->node2term_entries > I.cap_k1) return;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t node = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); node < I.N; node += warps) {
        const uint32_t nu = I.upper_count[node];
        const uint32_t ro = I.row_offset[node], re = I.row_offset[node + 1];
        const uint32_t h0 = I.half_offset[node];
        for (uint32_t u = lane_id(); u < nu; u += 32) {
            const uint32_t key = I.tmp_key[ro + u];
            const uint32_t start = I.tmp_start[ro + u];
            const uint32_t end = (u + 1 < nu) ? I.tmp_start[ro + u + 1] : re;
            I.half_key[h0 + u] = key;
            I.half_range[h0 + u] = make_uint2(start, end);
            atomicAdd(&I.lower_count[key % I.enc], 1u);
        }
    }
}

// warp per node: place the row's upper entries and scatter its pairs into the
// lower part of each partner row (unordered there; sorted next)
__global__ void __launch_bounds__(256) np_sym_scatter_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const DeviceCounts* C = I.counts;
    if (C->half_pairs > I.cap_pairs || C->nodepair_entries > I.cap_k2 || C->node2term_entries > I.cap_k1) return;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t node = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); node < I.N; node += warps) {
        const uint32_t nu = I.upper_count[node];
        const uint32_t h0 = I.half_offset[node];
        const uint32_t up0 = I.blkrow_offset[node] + I.lower_count[node];
        for (uint32_t u = lane_id(); u < nu; u += 32) {
            const uint32_t h = h0 + u;
            const uint32_t key = I.half_key[h];
            const uint2 rg = I.half_range[h];
            const uint32_t s = up0 + u;
            I.sym_key[s] = key;
            I.sym_range[s] = rg;
            I.sym_half[s] = h;
            const uint32_t j = key % I.enc;
            const uint32_t pos = I.blkrow_offset[j] + atomicAdd(&I.lower_cursor[j], 1u);
            I.sym_key[pos] = j * I.enc + node;
            I.sym_range[pos] = rg;
            I.sym_half[pos] = h;
        }
    }
}

// pair_order: the order in which the off-diagonal kernel takes the pairs, about
// longest first (that kernel lasts as long as its longest pairs). Each pair is
// summed by one thread, so the order leaves the results unchanged. A CTA sorts
// one window of consecutive pairs by entry count (a counting sort in shared
// memory); the windows' chunks of kPairChunk pairs are then dealt out in turn,
// all first chunks before all second ones. Atomics on global buckets for one
// order of all pairs cost 125 us on a 32,768-node instance (this: 4 us).
constexpr uint32_t kLenBuckets = 256;

__global__ void __launch_bounds__(kLenBuckets) pair_order_kernel(const InstDesc* insts) {
    chain_wait();
    constexpr uint32_t kPer = kPairWindow / kLenBuckets;
    __shared__ uint32_t count[kLenBuckets], warp_tot[kLenBuckets / 32], order[kPairWindow];
    const InstDesc& I = insts[blockIdx.y];
    const DeviceCounts* C = I.counts;
    if (C->half_pairs > I.cap_pairs || C->nodepair_entries > I.cap_k2 || C->node2term_entries > I.cap_k1) return;
    const uint32_t P = C->half_pairs, windows = pair_slots(P) / kPairWindow;
    for (uint32_t win = blockIdx.x; win < windows; win += gridDim.x) {
        const uint32_t base = win * kPairWindow;
        count[threadIdx.x] = 0;
        __syncthreads();
        uint32_t bucket[kPer], rank[kPer];
#pragma unroll
        for (uint32_t q = 0; q < kPer; ++q) {
            const uint32_t h = base + threadIdx.x + kLenBuckets * q;
            order[threadIdx.x + kLenBuckets * q] = kInvalid;
            bucket[q] = kLenBuckets;
            if (h >= P) continue;
            // four entries per bucket, so that the lengths up to 1020 are told apart
            const uint2 rg = I.half_range[h];
            bucket[q] = kLenBuckets - 1 - min((rg.y - rg.x) / 4, kLenBuckets - 1);
            rank[q] = atomicAdd(&count[bucket[q]], 1u);
        }
        __syncthreads();
        const uint32_t c = count[threadIdx.x], incl = warp_inclusive_scan(c);
        if (lane_id() == 31) warp_tot[threadIdx.x >> 5] = incl;
        __syncthreads();
        uint32_t before = 0;
        for (uint32_t w = 0; w < (threadIdx.x >> 5); ++w) before += warp_tot[w];
        count[threadIdx.x] = before + incl - c;
        __syncthreads();
#pragma unroll
        for (uint32_t q = 0; q < kPer; ++q)
            if (bucket[q] < kLenBuckets) order[count[bucket[q]] + rank[q]] = base + threadIdx.x + kLenBuckets * q;
        __syncthreads();
#pragma unroll
        for (uint32_t q = 0; q < kPer; ++q) {
            const uint32_t r = threadIdx.x + kLenBuckets * q;
            I.pair_order[(r / kPairChunk * windows + win) * kPairChunk + r % kPairChunk] = order[r];
        }
        __syncthreads();
    }
}

// warp per row: sort the lower part by key (keys are unique) by ranking
__global__ void __launch_bounds__(128) np_lower_sort_kernel(const InstDesc* insts) {
    chain_wait();
    constexpr uint32_t kMaxLower = 256;
    __shared__ uint32_t sk[4][kMaxLower];
    __shared__ uint2 sr[4][kMaxLower];
    __shared__ uint32_t sh[4][kMaxLower];
    const InstDesc& I = insts[blockIdx.y];
    const DeviceCounts* C = I.counts;
    if (C->half_pairs > I.cap_pairs || C->nodepair_entries > I.cap_k2 || C->node2term_entries > I.cap_k1) return;
    const uint32_t w = threadIdx.x >> 5;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t node = blockIdx.x * (blockDim.x >> 5) + w; node < I.N; node += warps) {
        const uint32_t nl = I.lower_count[node];
        const uint32_t b = I.blkrow_offset[node];
        if (nl > kMaxLower) {
            if (lane_id() == 0) set_error(I, kErrRowTooLong);
            continue;
        }
        for (uint32_t i = lane_id(); i < nl; i += 32) {
            sk[w][i] = I.sym_key[b + i];
            sr[w][i] = I.sym_range[b + i];
            sh[w][i] = I.sym_half[b + i];
        }
        __syncwarp();
        for (uint32_t i = lane_id(); i < nl; i += 32) {
            const uint32_t key = sk[w][i];
            uint32_t rank = 0;
            for (uint32_t m = 0; m < nl; ++m) rank += sk[w][m] < key ? 1u : 0u;
            I.sym_key[b + rank] = key;
            I.sym_range[b + rank] = sr[w][i];
            I.sym_half[b + rank] = sh[w][i];
        }
        __syncwarp();
        // column and half-storage position of every entry of this block row:
        // the diagonal first, then the row's symmetric keys (lower part sorted
        // above, upper part written by np_sym_scatter_kernel); pair h sits in
        // row min(i, j) at h + min(i, j) + 1
        const uint32_t ne = I.blkrow_offset[node + 1] - b, mask = I.enc - 1;
        for (uint32_t i = lane_id(); i <= ne; i += 32) {
            uint32_t col = node, pos = I.half_offset[node] + node;
            if (i > 0) {
                col = I.sym_key[b + i - 1] & mask;
                pos = I.sym_half[b + i - 1] + min(node, col) + 1;
                if (col < node) pos |= kTransposedBlock;
            }
            I.bsr_ent[b + node + i] = make_uint2(pos, col);
        }
        __syncwarp();
    }
}

// --------------------------------------------------- bin-block CSR -------
// computeBinLengthKernel (NodePairRowColumnIndex.cu:64-119), multi-CTA: the
// bin width is 6 x the longest block row (diagonal included) among the block
// rows that the bin's 32 scalar rows touch
__global__ void __launch_bounds__(256) bin_length_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const uint32_t nb = (6 * I.N + 31) / 32;
    if (blockIdx.x == 0 && threadIdx.x == 0) I.counts->num_bins = nb;
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b <= nb; b += gridDim.x * blockDim.x) {
        if (b == nb) { I.bin_scan[b] = 0; continue; }
        const uint32_t r0 = 32 * b / 6;
        uint32_t r1 = (32 * b + 31) / 6;
        r1 = min(r1, I.N - 1);
        uint32_t mx = 0;
        for (uint32_t r = r0; r <= r1; ++r) mx = max(mx, 1 + I.blkrow_offset[r + 1] - I.blkrow_offset[r]);
        I.bin_scan[b] = 32 * 6 * mx;
    }
}

// computeBinBlockedCSRRowPtrKernel (NodePairRowColumnIndex.cu:122-132) and the
// 0xFF fill of the column array (:273-281)
__global__ void __launch_bounds__(256) bin_rowptr_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const DeviceCounts* C = I.counts;
    const uint32_t nb = C->num_bins;
    if (C->binblock_nnz > I.cap_bb) return;
    const uint32_t ncol = C->binblock_nnz / 6;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 32 * (nb + 1); i += stride)
        I.bb_rowptr[i] = (int32_t)(i % 32 + I.bin_scan[i / 32]);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ncol; i += stride) I.bb_colptr[i] = -1;
}

// computeBinBlockedCSRColPtrKernel (NodePairRowColumnIndex.cu:136-179)
__global__ void __launch_bounds__(256) bin_colptr_kernel(const InstDesc* insts) {
    chain_wait();
    const InstDesc& I = insts[blockIdx.y];
    const DeviceCounts* C = I.counts;
    if (C->binblock_nnz > I.cap_bb || C->half_pairs > I.cap_pairs) return;
    const uint32_t rows = 6 * I.N;
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < rows; row += gridDim.x * blockDim.x) {
        const uint32_t br = row / 6, lane = row % 32;
        const uint32_t data = (uint32_t)(row % 32) + I.bin_scan[row / 32];
        uint32_t col = (data - lane) / 6 + lane;
        I.bb_colptr[col] = (int32_t)(6 * br);
        col += 32;
        for (uint32_t s = I.blkrow_offset[br]; s < I.blkrow_offset[br + 1]; ++s, col += 32)
            I.bb_colptr[col] = (int32_t)(6 * (I.sym_key[s] % I.enc));
    }
}

// ------------------------------------------------------------ launch -----

static inline dim3 grid2(uint32_t x, uint32_t B) { return dim3(x ? x : 1, B); }

cudaError_t set_index_smem_limits(size_t seg_bytes) {
    return cudaFuncSetAttribute(n2t_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)seg_bytes);
}

// A CTA per node in the row kernels, while there are few nodes, whose lists are long.
// Whole solves, us, with a warp / a CTA per node: 500 nodes 801 / 714, 800 2600 / 2417,
// 1,500 1845 / 1775, 2,200 1675 / 1600, 3,001 1571 / 1547, 4,096 1495 / 1500; 32,768 13705 /
// 13800, 16 x 4,096 10140 / 10470.
static bool wide_rows(const LaunchCfg& lc) { return (uint64_t)lc.B * lc.max_nodes < 4096; }

cudaError_t launch_build_index(const LaunchCfg& lc, InstDesc* d, cudaStream_t st) {
    const uint32_t B = lc.B;
    const uint32_t cpv = lc.chunks_per_view;
    const uint32_t spread = (uint32_t)lc.sm_count * 4;  // grid-stride kernels
    const bool chain = chain_kernels(lc);
    MVDR_LAUNCH(input_check_kernel, grid2(spread, B), 256, 0, st, d, lc.width, lc.height);
    // dense pixels
    MVDR_LAUNCH_IF_CHAINED(chain, compact_count_kernel<DensePred>, grid2(cpv * lc.max_views, B), 256, 0, st, d, lc.width, lc.height, cpv);
    MVDR_LAUNCH_IF_CHAINED(chain, compact_scan_kernel, grid2(1, B), 1024, 0, st, d, cpv, lc.max_views, 0);
    MVDR_LAUNCH_IF_CHAINED(chain, compact_write_kernel<DensePred>, grid2(cpv * lc.max_views, B), 256, 0, st, d, lc.width, lc.height, cpv, 0);
    // foreground pixels (the predicate is false when the term is off)
    MVDR_LAUNCH_IF_CHAINED(chain, compact_count_kernel<ForegroundPred>, grid2(cpv * lc.max_views, B), 256, 0, st, d, lc.width, lc.height, cpv);
    MVDR_LAUNCH_IF_CHAINED(chain, compact_scan_kernel, grid2(1, B), 1024, 0, st, d, cpv, lc.max_views, 1);
    MVDR_LAUNCH_IF_CHAINED(chain, compact_write_kernel<ForegroundPred>, grid2(cpv * lc.max_views, B), 256, 0, st, d, lc.width, lc.height, cpv, 1);
    MVDR_LAUNCH_IF_CHAINED(chain, prepare_pixels_kernel, grid2(spread, B), 256, 0, st, d, lc.precision == MVDR_PRECISION_MIXED);
    if (lc.max_tp) {
        MVDR_LAUNCH_IF_CHAINED(chain, feat_choose_kernel, grid2((lc.max_tp + 255) / 256, B), 256, 0, st, d);
        MVDR_LAUNCH_IF_CHAINED(chain, feat_compact_kernel, grid2(1, B), 1024, 0, st, d);
    }
    MVDR_LAUNCH_IF_CHAINED(chain, term_offsets_kernel, grid2(1, B), 32, 0, st, d);
    // node -> term
    MVDR_LAUNCH_IF_CHAINED(chain, n2t_count_kernel, grid2(spread, B), 256, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, node_scan_kernel, grid2(1, B), 1024, 0, st, d, (int)kScanN2T);
    MVDR_LAUNCH_IF_CHAINED(chain, n2t_scatter_kernel, grid2(spread, B), 256, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, n2t_warp_sort_kernel, grid2((lc.max_nodes + 7) / 8, B), 256, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, n2t_merge_sort_kernel, grid2(min(lc.max_nodes, (uint32_t)lc.sm_count * 12), B), 32 * kMergeWarps, 0, st, d);
    if (lc.cap_seg > kMergeMax)
        MVDR_LAUNCH_IF_CHAINED(chain, n2t_sort_kernel, grid2(min(lc.max_nodes, (uint32_t)lc.sm_count), B), 256, (size_t)lc.cap_seg * 4, st, d);
    // node pair -> term
    const bool wide = wide_rows(lc);
    const dim3 grow = grid2(wide ? lc.max_nodes : (lc.max_nodes + kRowWarps - 1) / kRowWarps, B);
    if (wide) MVDR_LAUNCH_IF_CHAINED(chain, np_row_count_kernel<kRowWarps>, grow, 32 * kRowWarps, 0, st, d);
    else MVDR_LAUNCH_IF_CHAINED(chain, np_row_count_kernel<1>, grow, 32 * kRowWarps, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, node_scan_kernel, grid2(1, B), 1024, 0, st, d, (int)kScanRows);
    if (wide) MVDR_LAUNCH_IF_CHAINED(chain, np_row_build_kernel<kRowWarps>, grow, 32 * kRowWarps, 0, st, d);
    else MVDR_LAUNCH_IF_CHAINED(chain, np_row_build_kernel<1>, grow, 32 * kRowWarps, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, node_scan_kernel, grid2(1, B), 1024, 0, st, d, (int)kScanUpper);
    MVDR_LAUNCH_IF_CHAINED(chain, np_half_compact_kernel, grid2((lc.max_nodes + 7) / 8, B), 256, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, node_scan_kernel, grid2(1, B), 1024, 0, st, d, (int)kScanBlkRows);
    MVDR_LAUNCH_IF_CHAINED(chain, np_sym_scatter_kernel, grid2((lc.max_nodes + 7) / 8, B), 256, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, np_lower_sort_kernel, grid2((lc.max_nodes + 3) / 4, B), 128, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, pair_order_kernel, grid2(min((lc.cap_pairs + kPairWindow - 1) / kPairWindow, spread), B), kLenBuckets, 0, st, d);
    // bin-block CSR structure
    MVDR_LAUNCH_IF_CHAINED(chain, bin_length_kernel, grid2((6 * lc.max_nodes / 32 + 256) / 256, B), 256, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, node_scan_kernel, grid2(1, B), 1024, 0, st, d, (int)kScanBins);
    MVDR_LAUNCH_IF_CHAINED(chain, bin_rowptr_kernel, grid2(spread, B), 256, 0, st, d);
    MVDR_LAUNCH_IF_CHAINED(chain, bin_colptr_kernel, grid2((6 * lc.max_nodes + 255) / 256, B), 256, 0, st, d);
    return cudaGetLastError();
}

}  // namespace mvdr
