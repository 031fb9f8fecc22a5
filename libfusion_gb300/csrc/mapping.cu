// mapping.cu -- block allocation, visible-block enumeration and TSDF/colour
// integration (src/voxel_hashing/depth_fusion.cu:15-575 and the hash core of
// src/data_struct/map_struct.cu:143-389).
//
// GB300 design, per frame and for every session of a batch:
//   import      (gbf_fuse) the caller's images and pose, and each pixel's
//               integration test and weight; a System frame has them from its ingest.
//   alloc       one thread per level-0 pixel walks the blocks of its truncation
//               band (3-D Bresenham, depth_fusion.cu:121-228); the CTA dedupes
//               the keys of its pixel tile in a shared-memory set and each
//               unique key is inserted once into the session's open-addressing
//               table with a 64-bit CAS (lock-free, no dropped blocks), stamping
//               the block with the fuse counter.
//   visible     (gbf_fuse; a frame has the list from its z-range pass) one thread
//               per ALLOCATED block (not per table slot): visible = stamped this
//               fuse OR a block corner projects into the image within
//               [zmin, zmax] (is_block_visible, depth_fusion.cu:15-47);
//               warp-aggregated append to the visible list.
//   integrate   one CTA per visible block (grid-stride), 4 voxels per thread,
//               coalesced SoA voxel read-modify-write; blocks allocated this
//               fuse skip the read and are written whole (lazy zeroing instead
//               of the reference's full-pool cudaMemset, map_struct.cu:90).
#include "gbf_device.cuh"
#include "gbf_kernels.h"
#include "gn_step.cuh"

namespace gbf {

namespace {

constexpr int kAllocThreads = 256;      // 32 pixels wide, 8 rows at a time
constexpr int kSetBits = 10, kSetSize = 1 << kSetBits;  // shared-memory key set per CTA

// Per-pixel part of the integration test and weight (update_map_with_colour_kernel,
// depth_fusion.cu:317-331, without normals; update_map_weighted_kernel, :390-405, with):
// every voxel projecting to a pixel shares them, so they are computed once per
// pixel.  System frames get the same values from level_maps_kernel.  (1e-2f lies
// just below the reference's double 1e-2: the floats below that are those below 1e-2f, and 1e-2f.)
__global__ void fuse_import_kernel(const SessionView *__restrict__ svs, FuseImport in, MapPose pose) {
    chain_begin();
    const SessionView &sv = svs[0];
    if (blockIdx.x == 0 && threadIdx.x < 32) store_map_pose(sv.ts, pose);
    const int W = sv.lv[0].w, H = sv.lv[0].h;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W * H) return;
    const int x = i % W, y = i / W;
    const float dist = reinterpret_cast<const float *>(reinterpret_cast<const char *>(in.depth) + y * in.depth_pitch)[x];
    sv.depth_raw[i] = dist;
    const uint8_t *px = in.rgb + y * in.rgb_pitch + (size_t)x * 3;
    sv.rgb4[i] = make_uchar4(px[0], px[1], px[2], 0);
    bool ok;
    float w;
    if (!in.nmap) {
        ok = !(isnan(dist) || dist <= 1e-2f || dist > sv.zmax_u || dist < sv.zmin_u);
        w = 1.0f / (dist * dist);
    } else {
        const float4 nc = reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(in.nmap) + y * in.nmap_pitch)[x];
        ok = !(isnan(dist) || isnan(nc.x) || dist > sv.zmax_u || dist < sv.zmin_u);
        w = fabsf(sinf(nc.z)) / (dist * dist);
    }
    sv.fuse_px[i] = make_float2(ok ? dist : __int_as_float(0x7fffffff), w);
}

// The blocks a CTA's pixels pass, each once: an open-addressed key set and the list of
// its entries.
struct BlockSet {
    __align__(16) unsigned long long key[kSetSize];
    unsigned long long list[kSetSize];
    int count;
};

// False when the set is full where the key belongs (caller inserts globally).  The entry
// is read before it is claimed: the pixels of a warp pass the same few blocks, whose keys
// are there already and are read at once, where a compare-and-swap takes one lane
// after the other.
__device__ __forceinline__ bool set_insert(BlockSet &set, unsigned long long key) {
    unsigned h = (unsigned)(key ^ (key >> 29) ^ (key >> 43)) * 0x9E3779B1u;
    unsigned s = h >> (32 - kSetBits);
    for (int p = 0; p < 64; ++p) {
        unsigned long long old = *static_cast<volatile unsigned long long *>(set.key + s);
        if (old == key) return true;
        if (old == kEmptyKey) {
            old = atomicCAS(set.key + s, kEmptyKey, key);
            if (old == key) return true;
            if (old == kEmptyKey) {
                set.list[atomicAdd(&set.count, 1)] = key;
                return true;
            }
        }
        s = (s + 1) & (kSetSize - 1);
    }
    return false;
}

__device__ __forceinline__ void visit_block(const SessionView &sv, BlockSet &set, int bx, int by, int bz, int frame) {
    if (!coord_ok(bx, by, bz)) {
        raise_flag(sv, GBF_FLAG_COORD_RANGE);
        return;
    }
    const unsigned long long key = pack_key(bx, by, bz);
    if (!set_insert(set, key)) insert_block(sv, key, bx, by, bz, frame);
}

// unproject_world (depth_fusion.cu:101-112) then worldPtToVoxelPos + voxelPosToBlockPos
__device__ __forceinline__ int3 pixel_block(const SessionView &sv, const M34 &T, int x, int y, float z) {
    const LevelK &K = sv.lv[0];
    const float px = (K.invfx * ((float)x - K.cx)) * z;
    const float py = (K.invfy * ((float)y - K.cy)) * z;
    const float3 w = T.apply(px, py, z);
    return make_int3(voxel_to_block(floor_ref(w.x / sv.voxel)), voxel_to_block(floor_ref(w.y / sv.voxel)),
                     voxel_to_block(floor_ref(w.z / sv.voxel)));
}

// The blocks within half the truncation of each valid pixel's depth, gathered per tile of
// 32 x 8 ROWS pixels and then looked up or created, a thread per block.  What bounded it
// was the way into the shared set, a 64-bit compare-and-swap per pixel and block with
// up to 32 lanes on one entry, and the set's own 8 KB cleared and scanned per 256 pixels;
// now it is the pixels' own arithmetic (64 sessions of 640x480, with the visible pass: 489
// -> 408 us entry read first, 353 two rows a thread, 302 four, 276 with the list).
template <int ROWS>
__global__ void __launch_bounds__(kAllocThreads) alloc_kernel(const SessionView *svs, int zrange_follows) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active) return;
    const int W = sv.lv[0].w, H = sv.lv[0].h;
    // a frame's z-range pass comes next; an update alone leaves the last raycast's grid and count
    if (zrange_follows) clear_zrange(sv, blockIdx.x * kAllocThreads + threadIdx.x, gridDim.x * kAllocThreads);
    const int tiles_x = (W + 31) / 32;
    const int x = (blockIdx.x % tiles_x) * 32 + (threadIdx.x & 31), y0 = (blockIdx.x / tiles_x) * (8 * ROWS);
    if (y0 >= H) return;  // uniform per CTA

    __shared__ BlockSet set;
    __shared__ M34 T;
    float zs[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        const int y = y0 + 8 * k + (threadIdx.x >> 5);
        zs[k] = x < W && y < H ? sv.depth_raw[(size_t)y * W + x] : __int_as_float(0x7fffffff);
    }
    for (int i = threadIdx.x; i < kSetSize / 2; i += kAllocThreads)
        reinterpret_cast<ulonglong2 *>(set.key)[i] = make_ulonglong2(kEmptyKey, kEmptyKey);
    if (threadIdx.x == 0) {
        T = load_m34(sv.ts->map_twc);
        set.count = 0;
    }
    __syncthreads();
    const int frame = sv.ctr[C_FRAME] + 1;  // counted by integrate_kernel
    if (blockIdx.x == 0 && threadIdx.x == 0) sv.ctr[C_NVIS] = 0;

#pragma unroll 1
    for (int k = 0; k < ROWS; ++k) {
        const int y = y0 + 8 * k + (threadIdx.x >> 5);
        float z = zs[0];
#pragma unroll
        for (int q = 1; q < ROWS; ++q) z = k == q ? zs[q] : z;
        // create_blocks_kernel (depth_fusion.cu:130-141)
        if (!(isnan(z) || z < sv.zmin_u || z > sv.zmax_u)) {
            const float z_thresh = sv.tau * 0.5f;
            const float z_near = fmaxf(sv.zmin_u, z - z_thresh);
            const float z_far = fminf(sv.zmax_u, z + z_thresh);
            if (z_near < z_far) {
                int3 bn = pixel_block(sv, T, x, y, z_near);
                const int3 bf = pixel_block(sv, T, x, y, z_far);
                const int3 d = make_int3(bf.x - bn.x, bf.y - bn.y, bf.z - bn.z);
                const int3 inc = make_int3(d.x < 0 ? -1 : 1, d.y < 0 ? -1 : 1, d.z < 0 ? -1 : 1);
                const int3 ab = make_int3(abs(d.x), abs(d.y), abs(d.z));
                const int3 e2 = make_int3(ab.x << 1, ab.y << 1, ab.z << 1);
                visit_block(sv, set, bn.x, bn.y, bn.z, frame);
                // Bresenham's line over block coordinates (depth_fusion.cu:153-227)
                if (ab.x >= ab.y && ab.x >= ab.z) {
                    int err1 = e2.y - 1, err2 = e2.z - 1;
                    for (int i = 0; i < ab.x; ++i) {
                        if (err1 > 0) { bn.y += inc.y; err1 -= e2.x; }
                        if (err2 > 0) { bn.z += inc.z; err2 -= e2.x; }
                        err1 += e2.y; err2 += e2.z; bn.x += inc.x;
                        visit_block(sv, set, bn.x, bn.y, bn.z, frame);
                    }
                } else if (ab.y >= ab.x && ab.y >= ab.z) {
                    int err1 = e2.x - 1, err2 = e2.z - 1;
                    for (int i = 0; i < ab.y; ++i) {
                        if (err1 > 0) { bn.x += inc.x; err1 -= e2.y; }
                        if (err2 > 0) { bn.z += inc.z; err2 -= e2.y; }
                        err1 += e2.x; err2 += e2.z; bn.y += inc.y;
                        visit_block(sv, set, bn.x, bn.y, bn.z, frame);
                    }
                } else {
                    int err1 = e2.y - 1, err2 = e2.x - 1;
                    for (int i = 0; i < ab.z; ++i) {
                        if (err1 > 0) { bn.y += inc.y; err1 -= e2.z; }
                        if (err2 > 0) { bn.x += inc.x; err2 -= e2.z; }
                        err1 += e2.y; err2 += e2.x; bn.z += inc.z;
                        visit_block(sv, set, bn.x, bn.y, bn.z, frame);
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < set.count; i += kAllocThreads) {
        const unsigned long long key = set.list[i];
        // unpack the 21-bit fields (sign-extend)
        const int bx = (int)((long long)(key << (64 - 3 * kCoordBits)) >> (64 - kCoordBits));
        const int by = (int)((long long)(key << (64 - 2 * kCoordBits)) >> (64 - kCoordBits));
        const int bz = (int)((long long)(key << (64 - kCoordBits)) >> (64 - kCoordBits));
        insert_block(sv, key, bx, by, bz, frame);
    }
}

// is_vertex_visible / is_block_visible (depth_fusion.cu:15-47)
__device__ __forceinline__ bool block_in_frustum(const SessionView &sv, const M34 &Tcw, int bx, int by, int bz) {
    const LevelK &K = sv.lv[0];
    const float scale = sv.block_metric;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int cx = bx + ((c & 1) ? 1 : 0), cy = by + ((c & 2) ? 1 : 0), cz = bz + ((c & 4) ? 1 : 0);
        const float3 p = Tcw.apply((float)cx * scale, (float)cy * scale, (float)cz * scale);
        const float u = (K.fx * p.x) / p.z + K.cx;
        const float v = (K.fy * p.y) / p.z + K.cy;
        if (!(u < 0 || v < 0 || u > (float)(K.w - 1) || v > (float)(K.h - 1) || p.z < sv.zmin_u || p.z > sv.zmax_u))
            return true;
    }
    return false;
}

// The visible blocks of a fuse without a raycast behind it (a frame makes its list with
// the raycast's z-range, zrange_kernel).
__global__ void __launch_bounds__(256, 6) visible_kernel(const SessionView *svs) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active) return;
    __shared__ M34 Tcw;
    if (threadIdx.x == 0) Tcw = load_m34(sv.ts->map_tcw);
    __syncthreads();
    const int frame = sv.ctr[C_FRAME] + 1;
    const int n = min(sv.ctr[C_NUSED], sv.pool);
    const int stride = gridDim.x * blockDim.x;
    // whole warps iterate together so the append stays warp-uniform
    for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const int id = base + threadIdx.x;
        bool vis = false;
        int tag = 0;
        if (id < n) {
            const int4 c = sv.bcoord[id];
            vis = sv.bstamp[id] == frame || block_in_frustum(sv, Tcw, c.x, c.y, c.z);
            tag = sv.bfresh[id] ? (int)0x80000000 : 0;
        }
        const int pos = warp_append(sv.ctr + C_NVIS, vis);
        if (vis) sv.vis[pos] = id | tag;
    }
}

constexpr int kIntThreads = 128;  // threads per integration CTA (512 / kIntThreads voxels each), 16 CTAs per SM

template <int LAYOUT>
__global__ void __launch_bounds__(kIntThreads, 16) integrate_kernel(const SessionView *__restrict__ svs) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active || sv.layout != LAYOUT) return;
    __shared__ M34 Tcw_s;
    if (threadIdx.x == 0) Tcw_s = load_m34(sv.ts->map_tcw);
    __syncthreads();
    // Everything the voxel loop reads from the session descriptor is copied to
    // registers first: the loop stores voxels through global pointers, which the
    // compiler would otherwise have to assume may alias the descriptor.
    const M34 Tcw = Tcw_s;
    const LevelK K = sv.lv[0];
    const int W = K.w, H = K.h;
    const int nvis = sv.ctr[C_NVIS];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sv.ts->integrated_blocks += nvis;
        sv.ctr[C_FRAME] += 1;  // the allocation stamp of this fuse; no kernel reads it beside this one
    }
    const float voxel = sv.voxel, tau = sv.tau, inv_tau = sv.inv_tau;
    const int *__restrict__ vis = sv.vis;
    const int4 *__restrict__ bcoord = sv.bcoord;
    const float2 *__restrict__ fuse_px = sv.fuse_px;
    const uchar4 *__restrict__ rgb4 = sv.rgb4;
    unsigned char *__restrict__ bfresh = sv.bfresh;
    void *__restrict__ vox_sw = sv.vox_sw;
    uchar4 *__restrict__ vox_rgb = sv.vox_rgb;

    for (int b = blockIdx.x; b < nvis; b += gridDim.x) {
        const int tagged = vis[b];
        const int id = tagged & 0x7fffffff;
        const bool fresh = tagged < 0;
        const int4 bc = bcoord[id];
#pragma unroll
        for (int half_i = 0; half_i < kBlockVoxels / kIntThreads; ++half_i) {
            const int li = threadIdx.x + half_i * kIntThreads;
            const int lx = li & 7, ly = (li >> 3) & 7, lz = li >> 6;
            const int vi = id * kBlockVoxels + li;
            const float3 p = Tcw.apply((float)(bc.x * 8 + lx) * voxel, (float)(bc.y * 8 + ly) * voxel,
                                       (float)(bc.z * 8 + lz) * voxel);
            const int u = __float2int_rd(((K.fx * p.x) / p.z + K.cx) + 0.5f);
            const int v = __float2int_rd(((K.fy * p.y) / p.z + K.cy) + 0.5f);
            bool upd = !(u < 0 || v < 0 || u > W - 1 || v > H - 1);
            float dist = 0.f, weight = 0.f, sdf = 0.f;
            if (upd) {
                // depth and weight of the pixel, rejected pixels as NaN (fuse_px)
                const float2 fp = fuse_px[v * W + u];
                dist = fp.x;
                weight = fp.y;
                upd = !isnan(dist);
            }
            if (upd) {
                sdf = dist - p.z;
                if (sdf < -tau) upd = false;
            }
            if (!upd) {
                if (fresh) {
                    store_sw_at<LAYOUT>(vox_sw, vi, 0.f, 0.f);
                    vox_rgb[vi] = make_uchar4(0, 0, 0, 0);
                }
                continue;
            }
            sdf = fminf(1.0f, sdf * inv_tau);
            Vox old;
            if (fresh) {
                old.sdf = 0.f; old.w = 0.f; old.rgb = make_uchar4(0, 0, 0, 0);
            } else {
                old = load_vox_at<LAYOUT>(vox_sw, vox_rgb, vi);
            }
            const uchar4 cn = rgb4[v * W + u];
            float nsdf, nw;
            uchar4 nrgb;
            if (old.w == 0.f) {
                nsdf = sdf; nw = weight; nrgb = cn;
            } else {
                // the four running means share one denominator: one correctly
                // rounded reciprocal, then each quotient by div_rn_by
                const float den = old.w + weight;
                const float rden = __frcp_rn(den);
                nsdf = div_rn_by(old.sdf * old.w + sdf * weight, den, rden);
                nw = old.w + weight;
                nrgb.x = (unsigned char)__float2int_rz(
                    div_rn_by((float)old.rgb.x * old.w + (float)cn.x * weight, den, rden));
                nrgb.y = (unsigned char)__float2int_rz(
                    div_rn_by((float)old.rgb.y * old.w + (float)cn.y * weight, den, rden));
                nrgb.z = (unsigned char)__float2int_rz(
                    div_rn_by((float)old.rgb.z * old.w + (float)cn.z * weight, den, rden));
                nrgb.w = 0;
            }
            store_sw_at<LAYOUT>(vox_sw, vi, nsdf, nw);
            vox_rgb[vi] = nrgb;
        }
        if (fresh && threadIdx.x == 0) bfresh[id] = 0;
    }
}

}  // namespace

void launch_fuse_import(const SessionView *d_sv, const Extent &ex, const FuseImport &in, const double pose[12],
                        cudaStream_t st) {
    const int n = ex.w * ex.h;
    MapPose p;
    for (int i = 0; i < 12; ++i) p.p[i] = pose[i];
    launch_kernel(fuse_import_kernel, (n + 255) / 256, 256, ex.chain, st, d_sv, in, p);
}

// CTAs per session of the visible-block pass (grid-stride over the allocated
// blocks, whose count only the device knows); enough for a pool's worth
// without launching a CTA per 256 pool slots
constexpr int kVisCtas = 152;

void launch_alloc(const SessionView *d_sv, int nslots, const Extent &ex, bool zrange_follows, cudaStream_t st) {
    // Rows of a thread: one where the image's CTAs then still start at once (8 per SM),
    // two up to four rounds of them, four beyond, where a block that several tiles see
    // costs more than the length of a CTA.  Allocation and visible pass in us with 1, 2, 4
    // rows: one 640x480 session 19.8, 20.4, 24.4; four 34.6, 32.8, 34.7; 64: 338, 300, 276.
    const auto alloc = [&](auto *kernel, int rows) {
        const dim3 g(((ex.w + 31) / 32) * ((ex.h + 8 * rows - 1) / (8 * rows)), nslots);
        launch_kernel(kernel, g, kAllocThreads, ex.chain, st, d_sv, zrange_follows ? 1 : 0);
    };
    const long long ctas = (long long)ex.w * ex.h / kAllocThreads * nslots;
    if (ctas <= 8 * 152) alloc(alloc_kernel<1>, 1);
    else if (ctas <= 4 * 8 * 152) alloc(alloc_kernel<2>, 2);
    else alloc(alloc_kernel<4>, 4);
}

void launch_integrate(const SessionView *d_sv, int nslots, const Extent &ex, const int *layouts, cudaStream_t st) {
    // One CTA per visible block, grid-stride.  16 CTAs of 128 threads are resident per
    // SM; a session alone takes twice as many, so that an SM done early finds
    // more (640x480, 5 mm: 88 us with 8 per SM, 73 with 16, 68 with 32, 66 with 64).
    // Many sessions fill the chip with 8 each, and a CTA's prologue then counts
    // (64 sessions: 1.77 ms with 8, 1.80 with 16, 1.88 with 32, 2.03 with 64).
    const int gi = 152 * max(8, 32 / nslots);
    const dim3 g(gi, nslots);
    if (layouts[GBF_VOXEL_REF]) launch_kernel(integrate_kernel<GBF_VOXEL_REF>, g, kIntThreads, ex.chain, st, d_sv);
    if (layouts[GBF_VOXEL_HALF]) launch_kernel(integrate_kernel<GBF_VOXEL_HALF>, g, kIntThreads, ex.chain, st, d_sv);
    if (layouts[GBF_VOXEL_SNORM]) launch_kernel(integrate_kernel<GBF_VOXEL_SNORM>, g, kIntThreads, ex.chain, st, d_sv);
}

void launch_fuse(const SessionView *d_sv, int nslots, const Extent &ex, const int *layouts, cudaStream_t st) {
    launch_alloc(d_sv, nslots, ex, false, st);
    const int gv = min(max((ex.max_pool + 255) / 256, 1), kVisCtas);
    launch_kernel(visible_kernel, dim3(gv, nslots), 256, ex.chain, st, d_sv);
    launch_integrate(d_sv, nslots, ex, layouts, st);
}

}  // namespace gbf
