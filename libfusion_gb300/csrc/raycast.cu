// raycast.cu -- z-range tiles and per-pixel raycast (src/voxel_hashing/
// ray_tracing.cu:63-425) plus the post-raycast pyramid (DeviceImage::
// resize_device_map, src/tracking/device_image.cpp:188-199).
//
// GB300 design:
//   begin     (raycast calls) the pose, the z-range grid (H/8 x W/8) to (100, 0); a
//             System frame has its pose from tracking and the grid cleared by the
//             allocation.
//   zrange    eight lanes per block: a visible block's screen box on the 1/8
//             grid and its depth interval (create_rendering_block, :63-126), then
//             integer atomicMin / atomicMax on the float bit patterns (all values
//             are positive) of every covered cell.  The reference's 16x16
//             rendering-tile list, its cudaMalloc and its host read-back
//             (:223-277) are gone; the union of its tiles is exactly the box.
//             In the same launch every allocated block marks the depth slices of
//             the cells that rays may meet it in, and gets the ids of its
//             neighbours at +x, +y, +z; a frame, and a raycast with visibility of
//             its own, make the visible list there too, before the integration.
//   raycast   one thread per pixel, 64-pixel CTAs (8x8 by default: a warp is
//             an 8x4 patch of one z-range cell);
//             the march of MapRenderingDelegate::operator() (:346-425), passing
//             slices without a block on the reference's own sample positions but
//             without looking, the block of the last sample kept, and a trilinear
//             read that spans blocks taking the others from the neighbour list.
//             Output: camera-frame float4 vertex (NaN = miss).
//             What bounds it: issue (a warp's lanes read, cross into other blocks
//             and interpolate at different steps), and for one session the longest
//             rays, some 250 steps of 0.5 us.  The slices are the same for all lanes of a
//             warp, so skipping them keeps the warp together, where skipping by
//             the unallocated block a ray is in (each lane its own) measured slower.
//             640x480, march: 64 sessions 4.10 -> 2.57 ms per tick (slices 3.60,
//             shorter sample code 3.34, neighbour lists 2.72, one interpolation path
//             per warp 2.57), one 0.193 -> 0.130; allocation, visible list, z-range,
//             slices and neighbours together 0.61 -> 0.47 and 0.040 -> 0.028 ms.
//   post      2x2 mean vertex pyramid, then normals of every level.
#include "gbf_device.cuh"
#include "gbf_kernels.h"
#include "gn_step.cuh"

namespace gbf {

namespace {

__global__ void ray_begin_kernel(const SessionView *__restrict__ svs, MapPose pose, int check_visibility) {
    chain_begin();
    const SessionView &sv = svs[0];
    if (blockIdx.x == 0 && threadIdx.x < 32) store_map_pose(sv.ts, pose);
    if (check_visibility && blockIdx.x == 0 && threadIdx.x == 32) sv.ctr[C_NVIS] = 0;  // counted again by zrange_kernel
    clear_zrange(sv, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// The depth slices of a cell that an allocated block may lie in: 64 slices of the
// raycast's depth range, the last one open-ended.  A ray whose sample lies in an
// empty slice of its cell samples no allocated block there, so the march may run
// through the slice without looking (raycast_kernel).  That has to hold for every
// block that a sample can fall in, visible or not: a block marks all cells within
// two pixels of its bounds and all slices of its depths, both widened by a margin
// above what a ray's positions stray by, and the whole image when it reaches the
// camera plane.
constexpr int kSlices = 64;
__device__ __forceinline__ float slice_scale(const SessionView &sv) { return (float)kSlices / (sv.zmax_r - sv.zmin_r); }

// How far (metres) a ray's sample may lie from the straight ray: a voxel, and the
// rounding of its positions.  A march adds at most N = its length in voxels
// steps to coordinates below A voxels, and each sum is off by at most half a
// unit in the last place, A 2^-23, the same way every time.
__device__ __forceinline__ float ray_margin(const SessionView &sv) {
    const LevelK &K = sv.lv[0];
    const float *t = sv.ts->map_twc;
    const float stretch = 1.f + fmaxf(fabsf(K.cx), fabsf((float)K.w - K.cx)) * K.invfx +
                          fmaxf(fabsf(K.cy), fabsf((float)K.h - K.cy)) * K.invfy;
    const float N = stretch * (fmaxf(sv.zmax_r, sv.zmax_u) + 4.f * sv.block_metric) * sv.inv_voxel;
    const float A = N + fmaxf(fabsf(t[3]), fmaxf(fabsf(t[7]), fabsf(t[11]))) * sv.inv_voxel;
    return sv.voxel * (1.f + N * (A * 0x1p-22f));
}

// The cells of a box, shared out to the eight lanes of a block.
template <class F>
__device__ __forceinline__ void for_cells(int x0, int y0, int x1, int y1, const F &f) {
    const int w = x1 - x0 + 1, n = w * (y1 - y0 + 1);
    const float inv = 1.0f / (float)w;
    for (int i = threadIdx.x & 7; i < n; i += 8) {
        // i / w: i + 1/2 keeps the quotient 1 / (2 w) clear of an integer, and w, n stay below 2^20
        const int row = (int)(((float)i + 0.5f) * inv);
        f(x0 + i - row * w, y0 + row);
    }
}

__device__ __forceinline__ float list_near(const SessionView &sv) {
    return sv.ctr[C_DEEP_SDF] ? __int_as_float(0xff800000) : sv.zmin_r - kListSdf * sv.tau;
}

// Whether a sample of a raycast at this pose, or the refined one of a hit, can lie in
// the block.  The refined sample lies before the one that found the hit by sdf x
// truncation, and so up to kListSdf truncations before the near plane (a fused sdf is
// never below -1; with an imported one that is, every block counts).  Only a
// block that a marched sample can meet marks slices.
// near: the depth from which blocks count (list_near).
__device__ __forceinline__ bool mark_slices(const SessionView &sv, const M34 &Tcw, float margin, float near,
                                            const int4 bc) {
    const LevelK &K = sv.lv[0];
    const float h = 0.5f * sv.block_metric;
    const float3 p = Tcw.apply(((float)bc.x + 0.5f) * sv.block_metric, ((float)bc.y + 0.5f) * sv.block_metric,
                               ((float)bc.z + 0.5f) * sv.block_metric);
    // half extents of the turned cube
    const float hx = h * (fabsf(Tcw.m[0]) + fabsf(Tcw.m[1]) + fabsf(Tcw.m[2])) + margin;
    const float hy = h * (fabsf(Tcw.m[4]) + fabsf(Tcw.m[5]) + fabsf(Tcw.m[6])) + margin;
    const float hz = h * (fabsf(Tcw.m[8]) + fabsf(Tcw.m[9]) + fabsf(Tcw.m[10])) + margin;
    const float z0 = p.z - hz, z1 = p.z + hz;
    if (!(z1 >= near)) return false;
    int cx0 = 0, cx1 = sv.zr_w - 1, cy0 = 0, cy1 = sv.zr_h - 1;
    if (z0 > 0.25f * sv.zmin_r) {
        const float i0 = 1.f / z0, i1 = 1.f / z1;
        const float xl = p.x - hx, xh = p.x + hx, yl = p.y - hy, yh = p.y + hy;
        const float ul = K.fx * (xl * (xl < 0.f ? i0 : i1)) + K.cx - 2.f, uh = K.fx * (xh * (xh < 0.f ? i1 : i0)) + K.cx + 2.f;
        const float vl = K.fy * (yl * (yl < 0.f ? i0 : i1)) + K.cy - 2.f, vh = K.fy * (yh * (yh < 0.f ? i1 : i0)) + K.cy + 2.f;
        if (uh < 0.f || vh < 0.f || ul > (float)K.w || vl > (float)K.h) return isinf(near);
        cx0 = max(0, (int)(ul * 0.125f));
        cx1 = min(cx1, (int)(uh * 0.125f));
        cy0 = max(0, (int)(vl * 0.125f));
        cy1 = min(cy1, (int)(vh * 0.125f));
    }
    if (!(z1 >= sv.zmin_r)) return true;
    const float scale = slice_scale(sv);
    const int s0 = min(max((int)((z0 - sv.zmin_r) * scale), 0), kSlices - 1);
    const int s1 = min((int)((z1 - sv.zmin_r) * scale), kSlices - 1);
    const unsigned long long bits = (~0ull >> (kSlices - 1 - (s1 - s0))) << s0;
    for_cells(cx0, cy0, cx1, cy1, [&](int x, int y) { atomicOr(sv.zr_slices + y * sv.zr_w + x, bits); });
    return true;
}

// A block's corner `c` in the camera frame and where it projects.
struct Corner {
    float3 p;
    float u, v;
};
__device__ __forceinline__ Corner block_corner(const SessionView &sv, const M34 &Tcw, const int4 bc, int c) {
    const LevelK &K = sv.lv[0];
    const int cx = bc.x + (c & 1), cy = bc.y + ((c >> 1) & 1), cz = bc.z + (c >> 2);
    Corner k;
    k.p = Tcw.apply((float)cx * sv.block_metric, (float)cy * sv.block_metric, (float)cz * sv.block_metric);
    k.u = (K.fx * k.p.x) / k.p.z + K.cx;
    k.v = (K.fy * k.p.y) / k.p.z + K.cy;
    return k;
}

// create_rendering_block (ray_tracing.cu:63-126) by eight lanes with a corner each, four
// blocks a warp (all lanes call): the block's screen box and depth interval into the grid.
__device__ __forceinline__ void mark_zrange(const SessionView &sv, const Corner &k, bool visible) {
    const float u = k.u / 8.0f, v = k.v / 8.0f;
    // the reference's running bounds from (zr_w, zr_h, -1, -1): a NaN coordinate changes none
    const float fu = floorf(u), fv = floorf(v), cu = ceilf(u), cv = ceilf(v);
    int ulx = (float)sv.zr_w > fu ? __float2int_rz(fu) : sv.zr_w, lrx = -1.f < cu ? __float2int_rz(cu) : -1;
    int uly = (float)sv.zr_h > fv ? __float2int_rz(fv) : sv.zr_h, lry = -1.f < cv ? __float2int_rz(cv) : -1;
    float zx = sv.zmax_r > k.p.z ? k.p.z : sv.zmax_r, zy = sv.zmin_r < k.p.z ? k.p.z : sv.zmin_r;
#pragma unroll
    for (int m = 1; m < 8; m <<= 1) {
        ulx = min(ulx, __shfl_xor_sync(0xffffffffu, ulx, m));
        uly = min(uly, __shfl_xor_sync(0xffffffffu, uly, m));
        lrx = max(lrx, __shfl_xor_sync(0xffffffffu, lrx, m));
        lry = max(lry, __shfl_xor_sync(0xffffffffu, lry, m));
        const float x = __shfl_xor_sync(0xffffffffu, zx, m), y = __shfl_xor_sync(0xffffffffu, zy, m);
        zx = fminf(zx, x);
        zy = fmaxf(zy, y);
    }
    ulx = max(ulx, 0);
    uly = max(uly, 0);
    lrx = min(lrx, sv.zr_w - 1);
    lry = min(lry, sv.zr_h - 1);
    zx = fmaxf(zx, sv.zmin_r);
    const bool renders = visible && ulx <= lrx && uly <= lry;  // (zy is never below zmin)
    const unsigned n = __ballot_sync(0xffffffffu, renders && (threadIdx.x & 7) == 0);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(sv.ctr + C_RENDER, __popc(n));
    if (renders) {
        const int ix = __float_as_int(zx), iy = __float_as_int(zy);
        for_cells(ulx, uly, lrx, lry, [&](int x, int y) {
            atomicMin(reinterpret_cast<int *>(sv.zr_min) + y * sv.zr_w + x, ix);
            atomicMax(reinterpret_cast<int *>(sv.zr_max) + y * sv.zr_w + x, iy);
        });
    }
    __syncwarp();
}

// The slices of an allocated block and, where rays may meet it, its neighbours' ids.
__device__ __forceinline__ void mark_block(const SessionView &sv, const M34 &Tcw, float margin, float near, const int4 bc,
                                           int id) {
    const int c = threadIdx.x & 7;
    if (mark_slices(sv, Tcw, margin, near, bc))
        sv.bnext[(size_t)id * 8 + c] =
            c == 0 ? id : find_block(sv, bc.x + (c & 1), bc.y + ((c >> 1) & 1), bc.z + (c >> 2));
}

// Eight lanes to a block, a corner, a share of the cells and a neighbour each:
// a session has some 20,000 blocks, which a thread each would leave to 600 warps
// of long loops.  LIST: the visible blocks are those of the list (a raycast after a
// fuse, from a pose of its own); the first half of the CTAs takes them, the second the
// allocated ones.  Otherwise the pass makes the list on its way, from every allocated
// block's corners, which are the ones the z-range projects (a visible pass ahead of
// this one took 7 us per 640x480 frame and 14 in a large map, a thread per block
// projecting its eight corners one after the other): visible = a corner in the image
// within [zmin, zmax] (is_block_visible, depth_fusion.cu:15-47; a raycast's own
// visibility, ray_tracing.cu:681-807) or, with TOUCHED, stamped by this fuse
// (check_visibility_flag_kernel's flag 2).
template <bool LIST, bool TOUCHED>
__global__ void __launch_bounds__(256, 6) zrange_kernel(const SessionView *__restrict__ svs) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active) return;
    __shared__ M34 Tcw;
    __shared__ float margin, near;
    if (threadIdx.x < 12) Tcw.m[threadIdx.x] = sv.ts->map_tcw[threadIdx.x];
    if (threadIdx.x == 32) margin = ray_margin(sv);
    if (threadIdx.x == 64) near = list_near(sv);
    __syncthreads();
    const int c = threadIdx.x & 7, per_cta = blockDim.x / 8, lists = LIST ? gridDim.x / 2 : 0;
    const int used = min(sv.ctr[C_NUSED], sv.pool);
    if (LIST && blockIdx.x < lists) {
        const int nvis = sv.ctr[C_NVIS];
        // whole warps iterate together: the corners meet by shuffles
        for (int base = blockIdx.x * per_cta + (threadIdx.x & ~31) / 8; base < nvis; base += lists * per_cta) {
            const int b = base + ((threadIdx.x & 31) >> 3);
            const int4 bc = sv.bcoord[sv.vis[min(b, nvis - 1)] & 0x7fffffff];
            mark_zrange(sv, block_corner(sv, Tcw, bc, c), b < nvis);
        }
        return;
    }
    const int first = (blockIdx.x - lists) * per_cta, stride = (gridDim.x - lists) * per_cta;
    if (LIST) {
        for (int id = first + threadIdx.x / 8; id < used; id += stride) mark_block(sv, Tcw, margin, near, sv.bcoord[id], id);
        return;
    }
    const int frame = sv.ctr[C_FRAME] + 1;
    const float umax = (float)(sv.lv[0].w - 1), vmax = (float)(sv.lv[0].h - 1);
    for (int base = first + (threadIdx.x & ~31) / 8; base < used; base += stride) {
        const int b = base + ((threadIdx.x & 31) >> 3), id = min(b, used - 1);
        const int4 bc = sv.bcoord[id];
        const Corner k = block_corner(sv, Tcw, bc, c);
        // is_vertex_visible: false comparisons (NaN) leave the corner in
        const bool in = !(k.u < 0 || k.v < 0 || k.u > umax || k.v > vmax || k.p.z < sv.zmin_u || k.p.z > sv.zmax_u);
        const unsigned corners = __ballot_sync(0xffffffffu, in) >> (threadIdx.x & 24) & 0xffu;
        const bool visible = b < used && (corners || (TOUCHED && sv.bstamp[id] == frame));
        const int pos = warp_append(sv.ctr + C_NVIS, visible && c == 0);
        if (visible && c == 0) sv.vis[pos] = id | (sv.bfresh[id] ? (int)0x80000000 : 0);
        mark_zrange(sv, k, visible);
        if (b < used) mark_block(sv, Tcw, margin, near, bc, id);
        __syncwarp();
    }
}

// sdf of pool voxel i (int32 index: the pool is validated to fit) and whether it
// has been observed (weight not 0).  Only the weight's zero test is needed, so the HALF
// and SNORM layouts test the binary16 weight bits instead of converting them.
template <int LAYOUT, class SV>
__device__ __forceinline__ float sdf_raw(const SV &sv, int i, bool &valid) {
    if (LAYOUT == GBF_VOXEL_REF) {
        const uint2 q = SV::load(reinterpret_cast<const uint2 *>(sv.vox_sw) + i);
        valid = __uint_as_float(q.y) != 0.f;
        return sdf_ref_unpack((short)(q.x & 0xffffu));
    } else {
        const unsigned q = SV::load(reinterpret_cast<const unsigned *>(sv.vox_sw) + i);
        valid = (q & 0x7fff0000u) != 0u;  // binary16 weight != +-0 (NaN counts as observed, as w != 0.f)
        return sdf_word_unpack<LAYOUT>((unsigned short)(q & 0xffffu));
    }
}

// Voxel (vx, vy, vz) of block id (looked up by the caller); not valid in an unallocated block (id < 0).
template <int LAYOUT, class SV>
__device__ __forceinline__ float vox_in(const SV &sv, int id, int vx, int vy, int vz, bool &valid) {
    valid = false;
    if (id < 0) return 0.f;
    return sdf_raw<LAYOUT>(sv, id * kBlockVoxels + (voxel_to_local(vz) * 64 + voxel_to_local(vy) * 8 + voxel_to_local(vx)),
                           valid);
}

// the trilinear sum in the order of read_sdf_interped (ray_tracing.cu:307-339)
__device__ __forceinline__ float trilinear(float fx, float fy, float fz, float c000, float c100, float c010, float c110,
                                           float c001, float c101, float c011, float c111) {
    const float gx = 1.0f - fx, gy = 1.0f - fy;
    const float r2 = gy * (gx * c000 + fx * c100) + fy * (gx * c010 + fx * c110);
    const float r3 = gy * (gx * c001 + fx * c101) + fy * (gx * c011 + fx * c111);
    return (1.0f - fz) * r2 + fz * r3;
}

// The trilinear read when the corners span two to eight blocks (about 1/3 of
// the reads): out of line, so that the march loop's code stays small.  i000:
// the block of corner (x0, y0, z0), looked up by the caller; the others from its
// neighbour list.
template <int LAYOUT, class SV>
__device__ __noinline__ float interp_spanning(const SV sv, int i000, int x0, int x1, int y0, int y1, int z0, int z1,
                                              float fx, float fy, float fz, bool &valid) {
    // corner k = (x, y, z bits) lies in the block of k's bits that step over a block face
    const int step = ((x1 >> 3) != (x0 >> 3) ? 1 : 0) | ((y1 >> 3) != (y0 >> 3) ? 2 : 0) | ((z1 >> 3) != (z0 >> 3) ? 4 : 0);
    const int *next = sv.bnext + (size_t)i000 * 8;
    const int i100 = SV::load(next + (1 & step)), i010 = SV::load(next + (2 & step)), i110 = SV::load(next + (3 & step));
    const int i001 = SV::load(next + (4 & step)), i101 = SV::load(next + (5 & step)), i011 = SV::load(next + (6 & step));
    const int i111 = SV::load(next + (7 & step));
    bool v0, v1, v2, v3, v4, v5, v6, v7;
    const float c000 = vox_in<LAYOUT>(sv, i000, x0, y0, z0, v0), c100 = vox_in<LAYOUT>(sv, i100, x1, y0, z0, v1);
    const float c010 = vox_in<LAYOUT>(sv, i010, x0, y1, z0, v2), c110 = vox_in<LAYOUT>(sv, i110, x1, y1, z0, v3);
    const float c001 = vox_in<LAYOUT>(sv, i001, x0, y0, z1, v4), c101 = vox_in<LAYOUT>(sv, i101, x1, y0, z1, v5);
    const float c011 = vox_in<LAYOUT>(sv, i011, x0, y1, z1, v6), c111 = vox_in<LAYOUT>(sv, i111, x1, y1, z1, v7);
    valid = v0 && v1 && v2 && v3 && v4 && v5 && v6 && v7;
    return trilinear(fx, fy, fz, c000, c100, c010, c110, c001, c101, c011, c111);
}

// True when `p` holds on every lane that runs this together (one asm: nothing can part
// the lanes between the two).  Which lanes do is up to the scheduler, so a result must
// not depend on it.
__device__ __forceinline__ bool all_converged(bool p) {
    unsigned all;
    asm volatile("{\n .reg .pred a, b;\n .reg .b32 m;\n setp.ne.u32 a, %1, 0;\n activemask.b32 m;\n"
                 " vote.sync.all.pred b, a, m;\n selp.u32 %0, 1, 0, b;\n}\n"
                 : "=r"(all)
                 : "r"((unsigned)p));
    return all != 0;
}

// read_sdf_interped (ray_tracing.cu:307-339) at a point whose floor (x0, y0, z0)
// and its block id are at hand; c000: the corner there, observed.  The reference reads the
// corners at pt + (0|1, 0|1, 0|1) and floors each sum: floor(p + 1) is floor(p) + 1
// unless p + 1 rounds up to the next integer, which a comparison tells.  When the
// eight corners lie in one block (about 2/3 of the samples) they are read by
// offset from it, all loads issued together -- unless a lane beside needs the spanning
// read, which then serves them all (the same eight voxels; a warp with both paid for both:
// march of 64 VGA sessions 2.73 -> 2.58 ms, the spanning read alone for all 2.70).  NaN
// unless all corners are observed (the reference's sum over NaN corners).
template <int LAYOUT, class SV>
__device__ __forceinline__ float read_sdf_interped(const SV &sv, int id, int li, float px, float py, float pz, int x0,
                                                   int y0, int z0, float c000, bool &valid) {
    const float qx = floorf(px), qy = floorf(py), qz = floorf(pz);
    const float fx = px - qx, fy = py - qy, fz = pz - qz;
    const bool plain = px + 1.0f < qx + 2.0f && py + 1.0f < qy + 2.0f && pz + 1.0f < qz + 2.0f;
    // li + 73 carries out of a 3-bit field where that coordinate is 7
    const bool inside = (((li + 73) ^ li ^ 73) & 0x248) == 0;
    float v;
    if (all_converged(plain && inside)) {
        const int i = id * kBlockVoxels + li;
        bool v1, v2, v3, v4, v5, v6, v7;
        const float c100 = sdf_raw<LAYOUT>(sv, i + 1, v1), c010 = sdf_raw<LAYOUT>(sv, i + 8, v2);
        const float c110 = sdf_raw<LAYOUT>(sv, i + 9, v3), c001 = sdf_raw<LAYOUT>(sv, i + 64, v4);
        const float c101 = sdf_raw<LAYOUT>(sv, i + 65, v5), c011 = sdf_raw<LAYOUT>(sv, i + 72, v6);
        const float c111 = sdf_raw<LAYOUT>(sv, i + 73, v7);
        v = trilinear(fx, fy, fz, c000, c100, c010, c110, c001, c101, c011, c111);
        valid = v1 && v2 && v3 && v4 && v5 && v6 && v7;
    } else {
        v = interp_spanning<LAYOUT>(sv, id, x0, floor_ref(px + 1.0f), y0, floor_ref(py + 1.0f), z0, floor_ref(pz + 1.0f),
                                    fx, fy, fz, valid);
    }
    return valid ? v : __int_as_float(0x7fffffff);
}

// The fields the march reads on every step, copied into registers once per
// thread: through the descriptor in global memory the compiler has to reload
// them (the same copy took the integration from 2.29 to 1.76 ms).  CHAINED: the launches
// before may still write what this one reads (chain_begin); a batch's are not, and read
// voxels and neighbours through the read-only path (a tick of 64 sessions 8.78 -> 8.73 ms).
template <bool CHAINED>
struct MarchView {
    template <class T>
    static __device__ __forceinline__ T load(const T *p) { return CHAINED ? *p : __ldg(p); }
    const HashSlot *table;
    const int *bnext;
    void *vox_sw;
    int cap, cap_mask, max_probe;
};

// One CTA marches a tile of kRayThreads pixels, tw wide and kRayThreads / tw
// high (tw = 4, 8, 16 or 32; the launch shape is a batch knob).  The default
// 8x8 tile gives each warp an 8x4 patch: coherent march lengths.
constexpr int kRayThreads = 64;
constexpr int kMaxMarch = 1 << 16;  // safety bound; the march advances >= 1 voxel per step

// RGB: also write the hits' voxel colours (a separate instantiation: the
// colour pointer kept live across the march costs the plain raycast spills).
template <int LAYOUT, bool RGB, bool CHAINED>
__global__ void __launch_bounds__(kRayThreads, 24) raycast_kernel(const SessionView *__restrict__ svs, float4 *vmap_ext,
                                                                  long long vmap_pitch, int tw, uint8_t *rgb_ext,
                                                                  long long rgb_pitch) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active || sv.layout != LAYOUT) return;
    // the reference skips the raycast when nothing was visible or renderable
    if (sv.ctr[C_NVIS] == 0 || sv.ctr[C_RENDER] == 0) return;
    const LevelK &K = sv.lv[0];
    const int th = kRayThreads / tw;
    const int tiles_x = (K.w + tw - 1) / tw;
    const int x = (blockIdx.x % tiles_x) * tw + (threadIdx.x % tw);
    const int y = (blockIdx.x / tiles_x) * th + (threadIdx.x / tw);
    __shared__ M34 Twc, Tcw;
    if (threadIdx.x == 0) {
        Tcw = load_m34(sv.ts->map_tcw);
        Twc = load_m34(sv.ts->map_twc);
    }
    __syncthreads();
    if (x >= K.w || y >= K.h) return;

    float4 *out = vmap_ext ? reinterpret_cast<float4 *>(reinterpret_cast<char *>(vmap_ext) + y * vmap_pitch) + x
                           : sv.vmap[sv.ts->idx][0] + (size_t)y * K.w + x;
    const float qnan = __int_as_float(0x7fffffff);
    *out = make_float4(qnan, qnan, qnan, qnan);
    // colour (raycast_with_colour, ray_tracing.cu:478-564): white unless a hit's
    // nearest voxel has been observed
    if (RGB) {
        uint8_t *px = rgb_ext + y * rgb_pitch + (long long)x * 3;
        px[0] = px[1] = px[2] = 255;
    }

    const int cx = __float2int_rd((float)x / 8), cy = __float2int_rd((float)y / 8);
    if (cx >= sv.zr_w || cy >= sv.zr_h) return;
    const float zr0 = sv.zr_min[cy * sv.zr_w + cx], zr1 = sv.zr_max[cy * sv.zr_w + cx];
    if ((double)zr1 < 1e-3 || (double)zr0 < 1e-3 || isnan(zr0) || isnan(zr1)) return;

    const float iv = sv.inv_voxel;
    // unproject (ray_tracing.cu:341-344): (x - cx) * invfx * z
    float ux = (((float)x - K.cx) * K.invfx) * zr0, uy = (((float)y - K.cy) * K.invfy) * zr0;
    float dist_s = norm3(ux, uy, zr0) * iv;
    float3 bs = Twc.apply(ux, uy, zr0);
    bs = make_float3(bs.x * iv, bs.y * iv, bs.z * iv);
    ux = (((float)x - K.cx) * K.invfx) * zr1;
    uy = (((float)y - K.cy) * K.invfy) * zr1;
    const float dist_e = norm3(ux, uy, zr1) * iv;
    float3 be = Twc.apply(ux, uy, zr1);
    be = make_float3(be.x * iv, be.y * iv, be.z * iv);
    float3 dir = make_float3(be.x - bs.x, be.y - bs.y, be.z - bs.z);
    const float dn = norm3(dir.x, dir.y, dir.z);
    dir = make_float3(dir.x / dn, dir.y / dn, dir.z / dn);
    float3 r = bs;

    const MarchView<CHAINED> mv{sv.table, sv.bnext, sv.vox_sw, sv.cap, sv.cap_mask, sv.max_probe};
    const float step_scale = sv.step_scale;
    // depth slice of a sample: (dist * z per dist - zmin) * slices per metre
    const unsigned long long slices = sv.zr_slices[cy * sv.zr_w + cx];
    const float slice_z = sv.zmin_r, slices_per_m = slice_scale(sv);
    const float z_per_dist = zr0 / dist_s;
    const float steps_per_slice = 1.0f / (2.0f * z_per_dist * slices_per_m);
    // the block of the last sample: consecutive samples usually stay in one.  (A per-CTA
    // shared-memory cache of block ids in front of the table measured slower.)
    int bx = 0x7fffffff, by = 0, bz = 0, id = -1;
    auto block_at = [&](int x, int y, int z) {
        if (x != bx || y != by || z != bz) {
            bx = x; by = y; bz = z;
            id = find_block(mv, x, y, z);
        }
    };
    float sdf = 1.0f, step;
    bool valid = false;
    for (int it = 0; dist_s < dist_e && it < kMaxMarch; ++it) {
        if (!valid) {
            // Outside any block the reference steps two voxels from sample to sample.
            // Through slices without a block the same positions are passed without
            // looking; with none ahead the ray misses.
            const float at = (dist_s * z_per_dist - slice_z) * slices_per_m;
            const int s = min(max((int)at, 0), kSlices - 1);
            const unsigned long long ahead = slices >> s;
            if (!(ahead & 1ull)) {
                if (!ahead) return;
                int n = (int)(((float)(s + __ffsll(ahead) - 1) - at) * steps_per_slice) + 1;
                do {
                    r = make_float3(r.x + dir.x * 2.0f, r.y + dir.y * 2.0f, r.z + dir.z * 2.0f);
                    dist_s += 2.0f;
                } while (--n > 0 && dist_s < dist_e);
                if (!(dist_s < dist_e)) return;
            }
        }
        // read_sdf (ray_tracing.cu:291-305): the voxel ToVector3i(pt).  (The reference also
        // stops where sdf turns positive after a negative one; a negative one stops it before.)
        const int vx = floor_ref(r.x), vy = floor_ref(r.y), vz = floor_ref(r.z);
        block_at(voxel_to_block(vx), voxel_to_block(vy), voxel_to_block(vz));
        sdf = qnan;
        valid = false;
        if (id >= 0) {
            const int li = voxel_to_local(vz) * 64 + voxel_to_local(vy) * 8 + voxel_to_local(vx);
            const float s = sdf_raw<LAYOUT>(mv, id * kBlockVoxels + li, valid);
            if (valid) sdf = s;
            if (sdf <= 0.5f && sdf >= -0.5f)
                sdf = read_sdf_interped<LAYOUT>(mv, id, li, r.x, r.y, r.z, vx, vy, vz, s, valid);
            if (sdf <= 0.0f) break;
        }
        step = valid ? fmaxf(sdf * step_scale, 1.0f) : 2.0f;
        r = make_float3(r.x + dir.x * step, r.y + dir.y * step, r.z + dir.z * step);
        dist_s += step;
    }
    bool found = false;
    if (sdf <= 0.0f) {
        step = sdf * step_scale;
        r = make_float3(r.x + dir.x * step, r.y + dir.y * step, r.z + dir.z * step);
        const int vx = floor_ref(r.x), vy = floor_ref(r.y), vz = floor_ref(r.z);
        block_at(voxel_to_block(vx), voxel_to_block(vy), voxel_to_block(vz));
        if (id >= 0) {
            const int li = voxel_to_local(vz) * 64 + voxel_to_local(vy) * 8 + voxel_to_local(vx);
            const float s = sdf_raw<LAYOUT>(mv, id * kBlockVoxels + li, found);
            if (found) {
                sdf = read_sdf_interped<LAYOUT>(mv, id, li, r.x, r.y, r.z, vx, vy, vz, s, found);
                step = sdf * step_scale;
                r = make_float3(r.x + dir.x * step, r.y + dir.y * step, r.z + dir.z * step);
            }
        }
    }
    if (found) {
        const float3 c = Tcw.apply(r.x * sv.voxel, r.y * sv.voxel, r.z * sv.voxel);
        *out = make_float4(c.x, c.y, c.z, 1.0f);
        if (RGB) {  // read_colour (ray_tracing.cu:427-441): the voxel ToVector3i(pt)
            const int vx = floor_ref(r.x), vy = floor_ref(r.y), vz = floor_ref(r.z);
            block_at(voxel_to_block(vx), voxel_to_block(vy), voxel_to_block(vz));
            if (id >= 0) {
                const int i = id * kBlockVoxels + (voxel_to_local(vz) * 64 + voxel_to_local(vy) * 8 + voxel_to_local(vx));
                bool observed;
                sdf_raw<LAYOUT>(mv, i, observed);
                if (observed) {
                    const uchar4 col = sv.vox_rgb[i];
                    uint8_t *px = rgb_ext + y * rgb_pitch + (long long)x * 3;
                    px[0] = col.x;
                    px[1] = col.y;
                    px[2] = col.z;
                }
            }
        }
    }
}

// cv::cuda::resize(vmap, 0.5): 2x2 mean of every channel
__global__ void vmap_down_kernel(const SessionView *__restrict__ svs, int level) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active || level >= sv.levels) return;
    const int w = sv.lv[level].w, h = sv.lv[level].h, pw = sv.lv[level - 1].w;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * h) return;
    const int x = i % w, y = i / w;
    const int set = sv.ts->idx;
    const float4 *s = sv.vmap[set][level - 1];
    const float4 a = s[(size_t)(2 * y) * pw + 2 * x], b = s[(size_t)(2 * y) * pw + 2 * x + 1];
    const float4 c = s[(size_t)(2 * y + 1) * pw + 2 * x], d = s[(size_t)(2 * y + 1) * pw + 2 * x + 1];
    sv.vmap[set][level][i] = make_float4((((a.x + b.x) + c.x) + d.x) * 0.25f, (((a.y + b.y) + c.y) + d.y) * 0.25f,
                                         (((a.z + b.z) + c.z) + d.z) * 0.25f, (((a.w + b.w) + c.w) + d.w) * 0.25f);
}

// computeNMapK (cuda_imgproc.cu:276-294) over every level of the reference set
// computeNMapK (cuda_imgproc.cu:276-305) at (x, y) of a vertex map whose rows are
// `stride` float4 apart: normalised cross product of the horizontal and vertical
// differences; NaN in the last row and column (written, where the reference
// leaves them unwritten) and wherever a neighbour is NaN.
template <class Get>
__device__ __forceinline__ float4 normal_by(const Get &V, int x, int y, int w, int h) {
    const float qnan = __int_as_float(0x7fffffff);
    if (x >= w - 1 || y >= h - 1) return make_float4(qnan, qnan, qnan, qnan);
    const int x10 = max(x - 1, 0), y10 = max(y - 1, 0);
    const float4 v00 = V(x10, y), v01 = V(x + 1, y);
    const float4 v10 = V(x, y10), v11 = V(x, y + 1);
    const float3 a = make_float3(v01.x - v00.x, v01.y - v00.y, v01.z - v00.z);
    const float3 bb = make_float3(v11.x - v10.x, v11.y - v10.y, v11.z - v10.z);
    const float3 n = cross3(a, bb);
    const float l = norm3(n.x, n.y, n.z);
    return make_float4(n.x / l, n.y / l, n.z / l, 1.f);
}
__device__ __forceinline__ float4 normal_at(const float4 *V, long long stride, int x, int y, int w, int h) {
    return normal_by([&](int xx, int yy) { return V[yy * stride + xx]; }, x, y, w, h);
}

// 2x2 mean of four vertices in vmap_down_kernel's order
__device__ __forceinline__ float4 mean4(const float4 a, const float4 b, const float4 c, const float4 d) {
    return make_float4((((a.x + b.x) + c.x) + d.x) * 0.25f, (((a.y + b.y) + c.y) + d.y) * 0.25f,
                       (((a.z + b.z) + c.z) + d.z) * 0.25f, (((a.w + b.w) + c.w) + d.w) * 0.25f);
}

// The post-raycast pyramid of up to three levels in one pass: a CTA takes a
// 32x32 tile of the level-0 vertex map with a 4-pixel halo into shared memory,
// writes the tile's level-0 normals, builds the 16x16 level-1 tile (2x2 means,
// vmap_down_kernel's arithmetic) with a 2-pixel halo and its normals, then the
// 8x8 level-2 tile with a 1-pixel halo and its normals -- the arithmetic of
// vmap_down_kernel and nmap_all_kernel, reading the level-0 map once instead of
// writing and re-reading every level.  The tile's loads all come first, a warp per row
// (in turn, with their coordinates divided out, they left a session's few CTAs waiting:
// 640x480 14.1 -> 12.5 us, four sessions 25.3 -> 22.6, 64 250 -> 242).
constexpr int kPostTile = 32;
__global__ void __launch_bounds__(256) post_pyramid_kernel(const SessionView *__restrict__ svs, unsigned *done,
                                                           unsigned number) {
    chain_begin();
    if (done && blockIdx.x == 0 && threadIdx.x == 0) *static_cast<volatile unsigned *>(done) = number;
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active) return;
    const int w0 = sv.lv[0].w, h0 = sv.lv[0].h;
    const int tiles_x = (w0 + kPostTile - 1) / kPostTile;
    const int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (ty * kPostTile >= h0) return;  // a smaller frame than the batch's largest
    const int set = sv.ts->idx;
    const float qnan = __int_as_float(0x7fffffff);
    const float4 nan4 = make_float4(qnan, qnan, qnan, qnan);
    __shared__ float4 s0[kPostTile + 8][kPostTile + 8];
    __shared__ float4 s1[kPostTile / 2 + 4][kPostTile / 2 + 4];
    __shared__ float4 s2[kPostTile / 4 + 2][kPostTile / 4 + 2];
    // level 0: the tile and its 4-pixel halo (outside the image: never read)
    const int ox0 = tx * kPostTile - 4, oy0 = ty * kPostTile - 4;
    const float4 *V0 = sv.vmap[set][0];
    // a warp per row: columns 0..31, then the eight that the halo adds, all loads first
    constexpr int kRows = (kPostTile + 8) / 8;
    {
        float4 a[kRows], b[kRows];
        const int xa = ox0 + lane, xb = ox0 + 32 + lane;
        const bool in_a = xa >= 0 && xa < w0, in_b = lane < 8 && xb < w0;
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const int y = oy0 + warp + 8 * k;
            const bool in = y >= 0 && y < h0;
            a[k] = b[k] = nan4;
            if (in && in_a) a[k] = V0[(size_t)y * w0 + xa];
            if (in && in_b) b[k] = V0[(size_t)y * w0 + xb];
        }
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            s0[warp + 8 * k][lane] = a[k];
            if (lane < 8) s0[warp + 8 * k][32 + lane] = b[k];
        }
    }
    __syncthreads();
    {
        const auto get0 = [&](int x, int y) { return s0[y - oy0][x - ox0]; };
        float4 *N0 = sv.nmap[set][0];
        const int x = tx * kPostTile + lane;
#pragma unroll
        for (int k = 0; k < kPostTile / 8; ++k) {
            const int y = ty * kPostTile + warp + 8 * k;
            if (x < w0 && y < h0) N0[(size_t)y * w0 + x] = normal_by(get0, x, y, w0, h0);
        }
    }
    if (sv.levels < 2) return;
    // level 1: the 16x16 tile and a 2-pixel halo, from the level-0 pixels in s0
    const int w1 = sv.lv[1].w, h1 = sv.lv[1].h;
    const int ox1 = tx * (kPostTile / 2) - 2, oy1 = ty * (kPostTile / 2) - 2;
    float4 *V1 = sv.vmap[set][1];
    for (int ly = warp; ly < kPostTile / 2 + 4 && lane < kPostTile / 2 + 4; ly += 8) {
        const int lx = lane, x = ox1 + lx, y = oy1 + ly;
        float4 v = nan4;
        if (x >= 0 && y >= 0 && x < w1 && y < h1) {
            // level-0 pixel (2x, 2y) sits at s0[2 ly][2 lx]
            v = mean4(s0[2 * ly][2 * lx], s0[2 * ly][2 * lx + 1], s0[2 * ly + 1][2 * lx], s0[2 * ly + 1][2 * lx + 1]);
            if (lx >= 2 && ly >= 2 && lx < kPostTile / 2 + 2 && ly < kPostTile / 2 + 2) V1[(size_t)y * w1 + x] = v;
        }
        s1[ly][lx] = v;
    }
    __syncthreads();
    {
        const auto get1 = [&](int x, int y) { return s1[y - oy1][x - ox1]; };
        float4 *N1 = sv.nmap[set][1];
        for (int i = threadIdx.x; i < (kPostTile / 2) * (kPostTile / 2); i += blockDim.x) {
            const int x = tx * (kPostTile / 2) + i % (kPostTile / 2), y = ty * (kPostTile / 2) + i / (kPostTile / 2);
            if (x < w1 && y < h1) N1[(size_t)y * w1 + x] = normal_by(get1, x, y, w1, h1);
        }
    }
    if (sv.levels < 3) return;
    // level 2: the 8x8 tile and a 1-pixel halo, from the level-1 pixels in s1
    const int w2 = sv.lv[2].w, h2 = sv.lv[2].h;
    const int ox2 = tx * (kPostTile / 4) - 1, oy2 = ty * (kPostTile / 4) - 1;
    float4 *V2 = sv.vmap[set][2];
    for (int i = threadIdx.x; i < (kPostTile / 4 + 2) * (kPostTile / 4 + 2); i += blockDim.x) {
        const int lx = i % (kPostTile / 4 + 2), ly = i / (kPostTile / 4 + 2), x = ox2 + lx, y = oy2 + ly;
        float4 v = nan4;
        if (x >= 0 && y >= 0 && x < w2 && y < h2) {
            // level-1 pixel (2x, 2y) sits at s1[2 ly][2 lx]
            v = mean4(s1[2 * ly][2 * lx], s1[2 * ly][2 * lx + 1], s1[2 * ly + 1][2 * lx], s1[2 * ly + 1][2 * lx + 1]);
            if (lx >= 1 && ly >= 1 && lx < kPostTile / 4 + 1 && ly < kPostTile / 4 + 1) V2[(size_t)y * w2 + x] = v;
        }
        s2[ly][lx] = v;
    }
    __syncthreads();
    const auto get2 = [&](int x, int y) { return s2[y - oy2][x - ox2]; };
    float4 *N2 = sv.nmap[set][2];
    for (int i = threadIdx.x; i < (kPostTile / 4) * (kPostTile / 4); i += blockDim.x) {
        const int x = tx * (kPostTile / 4) + i % (kPostTile / 4), y = ty * (kPostTile / 4) + i / (kPostTile / 4);
        if (x < w2 && y < h2) N2[(size_t)y * w2 + x] = normal_by(get2, x, y, w2, h2);
    }
}

__global__ void nmap_of_kernel(const float4 *vmap, long long vmap_pitch, float4 *nmap, long long nmap_pitch, int w,
                               int h) {
    chain_begin();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= w || y >= h) return;
    // the pitches are multiples of 16 bytes (checked by the caller)
    reinterpret_cast<float4 *>(reinterpret_cast<char *>(nmap) + y * nmap_pitch)[x] =
        normal_at(vmap, vmap_pitch / 16, x, y, w, h);
}

__global__ void nmap_all_kernel(const SessionView *__restrict__ svs, unsigned *done, unsigned number) {
    chain_begin();
    if (done && blockIdx.x == 0 && threadIdx.x == 0) *static_cast<volatile unsigned *>(done) = number;
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active) return;
    int b = blockIdx.x, level = 0;
    for (; level < sv.levels; ++level) {
        const int n = (sv.lv[level].w * sv.lv[level].h + blockDim.x - 1) / blockDim.x;
        if (b < n) break;
        b -= n;
    }
    if (level >= sv.levels) return;
    const int w = sv.lv[level].w, h = sv.lv[level].h;
    const int i = b * blockDim.x + threadIdx.x;
    if (i >= w * h) return;
    const int x = i % w, y = i / w;
    const int set = sv.ts->idx;
    sv.nmap[set][level][i] = normal_at(sv.vmap[set][level], w, x, y, w, h);
}

}  // namespace

// CTAs per session: six per SM, as many as are resident (an even number: with a
// list, half of them take it), fewer of many sessions, whose CTAs loop
static int zrange_ctas(const Extent &ex, int nslots) {
    return 2 * min(max((ex.max_pool + 31) / 32, 1), max(152, 152 * 3 / nslots));
}
void launch_zrange(const SessionView *d_sv, int nslots, const Extent &ex, ZrangeOf of, cudaStream_t st) {
    const dim3 g(zrange_ctas(ex, nslots), nslots);
    const auto go = [&](auto *kernel) { launch_kernel(kernel, g, 256, ex.chain, st, d_sv); };
    if (of == ZrangeOf::list) go(zrange_kernel<true, false>);
    else if (of == ZrangeOf::frustum) go(zrange_kernel<false, false>);
    else go(zrange_kernel<false, true>);
}

void launch_march(const SessionView *d_sv, int nslots, const Extent &ex, float4 *vmap_ext, long long vmap_pitch,
                  const int *layouts, cudaStream_t st, uint8_t *rgb_ext, long long rgb_pitch) {
    const int tw = ray_tile_width(ex), th = kRayThreads / tw;
    // every slot's tiles fit: a smaller frame has fewer tiles per row and per column
    const dim3 g(((ex.w + tw - 1) / tw) * ((ex.h + th - 1) / th), nslots);
    const auto march = [&](auto *kernel) {
        launch_kernel(kernel, g, kRayThreads, ex.chain, st, d_sv, vmap_ext, vmap_pitch, tw, rgb_ext, rgb_pitch);
    };
    if (rgb_ext) {
        if (layouts[GBF_VOXEL_REF]) march(raycast_kernel<GBF_VOXEL_REF, true, true>);
        if (layouts[GBF_VOXEL_HALF]) march(raycast_kernel<GBF_VOXEL_HALF, true, true>);
        if (layouts[GBF_VOXEL_SNORM]) march(raycast_kernel<GBF_VOXEL_SNORM, true, true>);
    } else if (ex.chain) {
        if (layouts[GBF_VOXEL_REF]) march(raycast_kernel<GBF_VOXEL_REF, false, true>);
        if (layouts[GBF_VOXEL_HALF]) march(raycast_kernel<GBF_VOXEL_HALF, false, true>);
        if (layouts[GBF_VOXEL_SNORM]) march(raycast_kernel<GBF_VOXEL_SNORM, false, true>);
    } else {
        if (layouts[GBF_VOXEL_REF]) march(raycast_kernel<GBF_VOXEL_REF, false, false>);
        if (layouts[GBF_VOXEL_HALF]) march(raycast_kernel<GBF_VOXEL_HALF, false, false>);
        if (layouts[GBF_VOXEL_SNORM]) march(raycast_kernel<GBF_VOXEL_SNORM, false, false>);
    }
}

void launch_nmap_of(const float4 *vmap, long long vmap_pitch, float4 *nmap, long long nmap_pitch, int w, int h,
                    cudaStream_t st) {
    launch_kernel(nmap_of_kernel, dim3((w + 127) / 128, h), 128, true, st, vmap, vmap_pitch, nmap, nmap_pitch, w, h);
}

int post_launches(const Extent &ex) { return ex.levels <= 3 ? 1 : ex.levels; }

void launch_post(const SessionView *d_sv, int nslots, const Extent &ex, unsigned *done, unsigned number, cudaStream_t st) {
    if (ex.levels <= 3) {
        const int tiles = ((ex.w + kPostTile - 1) / kPostTile) * ((ex.h + kPostTile - 1) / kPostTile);
        launch_kernel(post_pyramid_kernel, dim3(tiles, nslots), 256, ex.chain, st, d_sv, done, number);
        return;
    }
    int w = ex.w, h = ex.h, total = (w * h + 255) / 256;
    for (int l = 1; l < ex.levels; ++l) {
        w /= 2; h /= 2;
        launch_kernel(vmap_down_kernel, dim3((w * h + 255) / 256, nslots), 256, ex.chain, st, d_sv, l);
        total += (w * h + 255) / 256;
    }
    launch_kernel(nmap_all_kernel, dim3(total, nslots), 256, ex.chain, st, d_sv, done, number);
}

void launch_raycast(const SessionView *d_sv, const Extent &ex, const double pose[12], bool check_visibility,
                    float4 *vmap_ext, long long vmap_pitch, const int *layouts, cudaStream_t st, uint8_t *rgb_ext,
                    long long rgb_pitch) {
    MapPose p;
    for (int i = 0; i < 12; ++i) p.p[i] = pose[i];
    const int cells = (ex.w / 8) * (ex.h / 8);
    launch_kernel(ray_begin_kernel, (cells + 255) / 256, 256, ex.chain, st, d_sv, p, check_visibility ? 1 : 0);
    launch_zrange(d_sv, 1, ex, check_visibility ? ZrangeOf::frustum : ZrangeOf::list, st);
    launch_march(d_sv, 1, ex, vmap_ext, vmap_pitch, layouts, st, rgb_ext, rgb_pitch);
}

}  // namespace gbf
