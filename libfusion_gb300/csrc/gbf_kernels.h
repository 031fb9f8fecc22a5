// gbf_kernels.h -- host-side launchers of the sm_103a kernels.
//
// Every launcher takes the device array of SessionView for `nslots` slots and
// the largest image extent among them; slots whose `active` is 0 return at once.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/gbfusion.h"
#include "gbf_types.h"

namespace gbf {

struct Extent {
    int w, h;        // largest level-0 size among the slots
    int max_pool;    // largest block pool among the slots
    int max_red[kMaxLevels]; // largest reduction CTA count per level
    int levels;      // largest level count
    int max_iter[kMaxLevels];
    int ray_tw;      // raycast tile width (4, 8, 16 or 32 of a 64-pixel tile); 0 = 8
    int chain;       // 1: a session's own launches, one after the other on a stream (launch_kernel)
};

// A launch that, when chained, is set up while the launch before it in the stream
// still runs (programmatic dependent launch; the kernel waits in chain_begin).  A frame
// of one session is a chain of a dozen launches of 4 to 150 us, with 2.0 to 2.5 us between two
// plain ones and 0.4 between chained ones.  A batch's ticks launch plainly: captured,
// their launches are 0.5 us apart, and the CTAs that wait early would take the places of the
// other branch's.
template <class... P, class... A>
inline void launch_kernel(void (*kernel)(P...), dim3 grid, int threads, bool chain, cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = chain ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, P(args)...);
}

inline int ray_tile_width(const Extent &ex) {
    return (ex.ray_tw == 4 || ex.ray_tw == 16 || ex.ray_tw == 32) ? ex.ray_tw : 8;
}

// ---- ingest (ingest.cu) ------------------------------------------------------
struct IngestArgs {
    int set_sel;                 // 0: current set (1-idx), 1: reference set (idx)
    int src;                     // 0: staging u16+rgb8, 1: external u16, 2: external float
    const void *depth; long long depth_pitch;
    const uint8_t *rgb; long long rgb_pitch;
};
// kernel launches of one launch_ingest
inline int ingest_launches(const Extent &ex) { return 2 + (ex.levels > 3 ? ex.levels - 3 : 0); }
void launch_ingest(const SessionView *d_sv, int nslots, const Extent &ex, const IngestArgs &a, cudaStream_t st);

// ---- mapping (mapping.cu) ------------------------------------------------------
struct FuseImport {
    const float *depth; long long depth_pitch;
    const uint8_t *rgb; long long rgb_pitch;
    const float *nmap; long long nmap_pitch;
};
// the caller's images and pose: colour update (1/d^2), or weighted with the imported normals
void launch_fuse_import(const SessionView *d_sv, const Extent &ex, const FuseImport &in, const double pose[12],
                        cudaStream_t st);
void launch_fuse(const SessionView *d_sv, int nslots, const Extent &ex, const int *layouts, cudaStream_t st);
// the blocks of the frame's surface; also clears the visible count and, for a z-range
// pass that follows, its grid
void launch_alloc(const SessionView *d_sv, int nslots, const Extent &ex, bool zrange_follows, cudaStream_t st);
// Phong shading of camera-frame vertex / normal maps into RGBA8 (rgb NULL = untextured)
void launch_render(const float4 *vmap, long long vmap_pitch, const float4 *nmap, long long nmap_pitch,
                   const uint8_t *rgb, long long rgb_pitch, int rgb_stride, int w, int h, uchar4 *out,
                   long long out_pitch, cudaStream_t st);
void launch_integrate(const SessionView *d_sv, int nslots, const Extent &ex, const int *layouts, cudaStream_t st);
// the session's model prediction, shaded (textured: with the last frame's colour)
void launch_render_session(const SessionView *d_sv, const Extent &ex, int textured, uchar4 *out, long long out_pitch,
                           cudaStream_t st);

// ---- raycast (raycast.cu) -------------------------------------------------------
// One session's raycast at `pose`, optionally over the visible blocks of that pose.
// rgb_ext (optional): the hits' nearest voxel colours, 3 bytes per pixel, white elsewhere
void launch_raycast(const SessionView *d_sv, const Extent &ex, const double pose[12], bool check_visibility,
                    float4 *vmap_ext, long long vmap_pitch, const int *layouts, cudaStream_t st,
                    uint8_t *rgb_ext = nullptr, long long rgb_pitch = 0);
// The z-range pass, its grid cleared before (launch_alloc, launch_raycast): of the visible
// list, or making the list on its way -- the blocks in the frustum of the map pose, or
// those and the ones that this fuse touched.
enum class ZrangeOf { list, frustum, fuse };
void launch_zrange(const SessionView *d_sv, int nslots, const Extent &ex, ZrangeOf of, cudaStream_t st);
void launch_march(const SessionView *d_sv, int nslots, const Extent &ex, float4 *vmap_ext, long long vmap_pitch,
                  const int *layouts, cudaStream_t st, uint8_t *rgb_ext = nullptr, long long rgb_pitch = 0);
// computeNMapK (cuda_imgproc.cu:276-305) of a pitched vertex map into a pitched normal map
void launch_nmap_of(const float4 *vmap, long long vmap_pitch, float4 *nmap, long long nmap_pitch, int w, int h,
                    cudaStream_t st);
// kernel launches of one launch_post
int post_launches(const Extent &ex);
// done (optional): where the frame's number is noted as it ends
void launch_post(const SessionView *d_sv, int nslots, const Extent &ex, unsigned *done, unsigned number, cudaStream_t st);

// The ICP gates sine < angle and length <= dist (pose_estimator.cu:200) as bounds on
// the squares whose rounded roots they compare: the root rounded to nearest is
// monotonic, so exactly the squares below angle2, and those up to dist2, pass.  The
// two roots per pixel and iteration cost 2.5% of a 64-session tracking phase.
inline void square_gates(SessionView &v, float dist, float angle) {
    float a = angle > 0.f ? angle * angle : 0.f;  // the least float whose root is not below angle
    while (a > 0.f && sqrtf(nextafterf(a, 0.f)) >= angle) a = nextafterf(a, 0.f);
    while (a < INFINITY && sqrtf(a) < angle) a = nextafterf(a, INFINITY);
    float d = dist >= 0.f ? dist * dist : -1.f;  // the greatest float whose root is not above dist
    while (d > 0.f && sqrtf(d) > dist) d = nextafterf(d, 0.f);
    while (d >= 0.f && d < INFINITY && sqrtf(nextafterf(d, INFINITY)) <= dist) d = nextafterf(d, INFINITY);
    v.icp_angle2 = a;
    v.icp_dist2 = d;
}

// ---- tracking (tracking.cu) -----------------------------------------------------
// mode 0: full Gauss-Newton (gbf_track / process frame), stops at the schedule end
// alone: little of this library's work runs beside it (not one of several branches of a
// tick, nor one of several streams' frames), so a few sessions may take the whole chip.
// kernel launches of one launch_track over nslots sessions
int track_launches(int nslots, const Extent &ex, bool alone);
void launch_track(const SessionView *d_sv, int nslots, const Extent &ex, int frame_mode, bool alone, cudaStream_t st);
// whether a launch of these sessions alone on the chip tracks in one run
bool track_run_fits(int nslots, const Extent &ex);
// what launch_track needs of the current device, asked once (before any stream capture)
void prepare_track();
// single reduction for gbf_reduce: pose given as float 3x4 in the kernel args
void launch_reduce_once(const SessionView *d_sv, const Extent &ex, int level, const float *pose12, float stddev,
                        cudaStream_t st);
// frame bookkeeping after tracking: pose update, reference swap
void launch_frame_finish(const SessionView *d_sv, int nslots, cudaStream_t st);
// per-slot pose / tracking / status record of a batch tick (empty slots zero)
void launch_slot_results(const SessionView *d_sv, int nslots, gbf_slot_result *out, cudaStream_t st);

// ---- meshing (mesh.cu) ------------------------------------------------------------
// returns via device counters; the host reads C_MESH_TRIS.  counts, chunk_sums: the session's mesh_off and mesh_sums
void launch_mesh(const SessionView *d_sv, const Extent &ex, int layout, int mode, float *vtx, void *attr,
                 long long max_tris, int *counts, int *chunk_sums, cudaStream_t st);

}  // namespace gbf
