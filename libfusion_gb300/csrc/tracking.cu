// tracking.cu -- fused point-to-plane ICP + photometric normal equations and
// the device-side Gauss-Newton step (src/tracking/pose_estimator.cu:166-307,
// src/tracking/m_estimator.cu:313-482, include/tracking/reduce_sum.h:11-61,
// src/tracking/icp_tracker.cpp:23-156).
//
// GB300 design: one launch per (level, iteration) for all sessions of a batch.
// Each CTA reduces its pixels' ICP row and photometric row (the reference runs
// two kernels, each re-reading the reference vertex map) into 29 + 29 FP32
// sums (warp shuffle tree, then a fixed-order shared-memory pass), writes one
// partial record, and the last CTA of the session (atomic ticket) adds the
// partials in a fixed order by compensated float addition, then its first warp
// runs the step on the device: FP64 LDL^T solve of the 6x6 system, SE(3)
// exponential, pose composition, and the reference's error-increase / revert /
// break rules.  Launches of 32 or more sessions take the sum and the step in a
// launch of their own (one CTA per session) instead, so that the reduction's
// CTAs end without a fence and a ticket; the sums and the step are the same.
// No host round trip: the reference pays two device->host syncs per iteration
// (pose_estimator.cu:302-304, m_estimator.cu:477-479).  The order of every sum is fixed, so a session's
// result does not depend on the other sessions in the batch.
#include <float.h>
#include <string.h>

#include <atomic>
#include <mutex>

#include "gbf_device.cuh"
#include "gbf_internal.h"
#include "gbf_kernels.h"
#include "gn_step.cuh"

namespace gbf {

namespace {

// |log(T)| of an SE(3) element (the success test, icp_tracker.cpp:145)
__device__ double se3_log_norm(const double T[12]) {
    const double tr = T[0] + T[5] + T[10];
    double c = (tr - 1.0) * 0.5;
    c = c > 1.0 ? 1.0 : (c < -1.0 ? -1.0 : c);
    const double th = acos(c);
    const double vx = T[9] - T[6], vy = T[2] - T[8], vz = T[4] - T[1];
    double k = 0.5;
    const double s = sin(th);
    if (th > 1e-8 && s > 1e-12) k = th / (2.0 * s);
    const double wx = k * vx, wy = k * vy, wz = k * vz;
    // rho = V^-1 t,  V^-1 = I - W/2 + (1/th^2)(1 - A/(2B)) W^2
    const double th2 = wx * wx + wy * wy + wz * wz;
    double f;
    if (th2 < 1e-10) {
        f = 1.0 / 12.0;
    } else {
        const double t = sqrt(th2);
        const double A = sin(t) / t, B = (1.0 - cos(t)) / th2;
        f = (1.0 - A / (2.0 * B)) / th2;
    }
    const double W[9] = {0, -wz, wy, wz, 0, -wx, -wy, wx, 0};
    const double t3[3] = {T[3], T[7], T[11]};
    double rho[3];
    for (int i = 0; i < 3; ++i) {
        double r = t3[i];
        for (int j = 0; j < 3; ++j) {
            double w2 = W[i * 3] * W[j] + W[i * 3 + 1] * W[3 + j] + W[i * 3 + 2] * W[6 + j];
            r += -0.5 * W[i * 3 + j] * t3[j] + f * w2 * t3[j];
        }
        rho[i] = r;
    }
    return sqrt(rho[0] * rho[0] + rho[1] * rho[1] + rho[2] * rho[2] + th2);
}

// ---------------------------------------------------------------------------
// per-pixel rows
__device__ __forceinline__ float interp2(const float *img, int w, float x, float y) {
    const int u = (int)floorf(x), v = (int)floorf(y);
    const float ax = x - (float)u, ay = y - (float)v;
    const float *r0 = img + (size_t)v * w, *r1 = r0 + w;
    return (r0[u] * (1.0f - ax) + r0[u + 1] * ax) * (1.0f - ay) + (r1[u] * (1.0f - ax) + r1[u + 1] * ax) * ay;
}

// interp2 of the intensity and both gradients at once from the packed
// (I, dI/dx, dI/dy, 0) image: four 16-byte taps, each channel the same
// expression as interp2.
__device__ __forceinline__ float3 interp2_igd(const float4 *img, int w, float x, float y) {
    const int u = (int)floorf(x), v = (int)floorf(y);
    const float ax = x - (float)u, ay = y - (float)v;
    const float4 *r0 = img + (size_t)v * w, *r1 = r0 + w;
    const float4 a = r0[u], b = r0[u + 1], c = r1[u], d = r1[u + 1];
    const float bx = 1.0f - ax, by = 1.0f - ay;
    return make_float3((a.x * bx + b.x * ax) * by + (c.x * bx + d.x * ax) * ay,
                       (a.y * bx + b.y * ax) * by + (c.y * bx + d.y * ax) * ay,
                       (a.z * bx + b.z * ax) * by + (c.z * bx + d.z * ax) * ay);
}

// What the rows of one level read besides the reference pixel.
struct LevelIn {
    int w, h;
    float fx, fy, cx, cy;
    float angle2, dist2;                  // the ICP gates, on squared lengths
    const float4 *__restrict__ vcur, *__restrict__ ncur, *__restrict__ igd;  // current frame
};
__device__ __forceinline__ LevelIn level_in(const SessionView &sv, int level, int cs) {
    const LevelK &K = sv.lv[level];
    return LevelIn{K.w, K.h, K.fx, K.fy, K.cx, K.cy, sv.icp_angle2, sv.icp_dist2,
                   sv.vmap[cs][level], sv.nmap[cs][level], sv.igd[cs][level]};
}

// ICPReduction::searchPoint + getRow (pose_estimator.cu:168-222)
__device__ __forceinline__ bool icp_row(const LevelIn &K, const M34 &T, const float4 vl, const float4 nl4,
                                        float row[7]) {
    if (isnan(vl.x)) return false;
    const float3 vg = T.apply(vl.x, vl.y, vl.z);
    // float invz = 1.0 / vlast_g.z in the reference: a double division rounded to
    // float.  For a float z that equals the correctly rounded float reciprocal
    // (1/z lies at least 2^-49 relative from any 25-bit rounding midpoint, so
    // the double rounding cannot change it), computed without FP64 hardware.
    const float invz = __frcp_rn(vg.z);
    const int u = __float2int_rd(((vg.x * invz) * K.fx + K.cx) + 0.5f);
    const int v = __float2int_rd(((vg.y * invz) * K.fy + K.cy) + 0.5f);
    if (u < 0 || v < 0 || u >= K.w || v >= K.h) return false;
    const int q = v * K.w + u;
    const float4 vc4 = K.vcur[q];
    const float3 ng = T.rotate(nl4.x, nl4.y, nl4.z);
    const float4 nc4 = K.ncur[q];
    const float dist2 = norm3_sq(vg.x - vc4.x, vg.y - vc4.y, vg.z - vc4.z);
    const float3 cr = cross3(make_float3(nc4.x, nc4.y, nc4.z), ng);
    const float sine2 = norm3_sq(cr.x, cr.y, cr.z);
    if (!(sine2 < K.angle2 && dist2 <= K.dist2 && !isnan(nc4.x) && !isnan(ng.x))) return false;
    const float3 vxn = cross3(vg, ng);
    row[0] = ng.x; row[1] = ng.y; row[2] = ng.z;
    row[3] = vxn.x; row[4] = vxn.y; row[5] = vxn.z;
    row[6] = dot3(ng, make_float3(vc4.x - vg.x, vc4.y - vg.y, vc4.z - vg.z));
    return true;
}

// Photometric constants of one reduction (m_estimator.cu:366-373).  The
// reference compares and scales in double; each FP64 instruction of a warp holds
// its quarter of the SM for 64 cycles, so the comparisons use the floats that
// divide at the same place (1e-4f and 1e-5f lie just below 1e-4 and 1e-5), and
// one thread of a CTA makes the product (photo_huber).
struct PhotoConst {
    float stddev, huber;
    float div, inv;  // res / stddev as div_rn_by(res, div, inv)
    bool normalise, robust;
};
__device__ __forceinline__ float photo_huber(float stddev) { return (float)(1.345 * (double)stddev); }
__device__ __forceinline__ PhotoConst photo_const(float stddev, float huber) {
    PhotoConst c;
    c.stddev = stddev;
    // six rows leave stddev infinite and the residuals zero: 0 * res, remainder res,
    // where an infinite div would make the remainder NaN
    c.inv = __frcp_rn(stddev);
    c.div = isinf(stddev) ? 0.f : stddev;
    c.normalise = stddev > 1e-4f;
    c.robust = stddev > 1e-5f;
    c.huber = huber;
    return c;
}

// RgbReduction2::find_corresp + compute_jacobian (m_estimator.cu:315-391).
// PACKED: the current frame's intensity and gradients from its packed image
// (sessions); otherwise from the three separate images (caller-owned images).
template <bool PACKED>
__device__ __forceinline__ bool rgb_row(const SessionView &sv, int level, int cs, const LevelIn &K, const M34 &T,
                                        const PhotoConst &pc, const float4 pt, const float il, float row[7]) {
    const float stddev = pc.stddev;
    if (pt.w < 0 || isnan(pt.x)) return false;
    if (!isfinite(il)) return false;
    const float3 q = T.apply(pt.x, pt.y, pt.z);
    // float z_inv = 1.0 / z (same argument as icp_row).  Sessions divide by it (div_rn_by:
    // 2.984 -> 2.946 ms over the tracking phase of 64; the residual's quotient by 1 / stddev
    // gave 0.03 ms away again); a caller's images may hold any z and divide.
    const float zi = __frcp_rn(q.z);
    const float u0 = (PACKED ? div_rn_by(q.x, q.z, zi) : q.x / q.z) * K.fx + K.cx;
    const float v0 = (PACKED ? div_rn_by(q.y, q.z, zi) : q.y / q.z) * K.fy + K.cy;
    if (!(u0 >= 2 && u0 < (float)(K.w - 2) && v0 >= 2 && v0 < (float)(K.h - 2))) return false;
    float ic, dx, dy;
    if (PACKED) {
        const float3 g = interp2_igd(K.igd, K.w, u0, v0);
        ic = g.x;
        dx = g.y;
        dy = g.z;
    } else {
        ic = interp2(sv.inten[cs][level], K.w, u0, v0);
        dx = interp2(sv.gx[level], K.w, u0, v0);
        dy = interp2(sv.gy[level], K.w, u0, v0);
    }
    if (!((dx > 2 || dy > 2) && isfinite(ic) && isfinite(dx) && isfinite(dy))) return false;
    const float lx = (dx * K.fx) * zi, ly = (dy * K.fy) * zi;
    const float lz = (-(lx * q.x + ly * q.y)) * zi;
    float res = ic - il;
    if (pc.normalise) res /= stddev;
    const float huber = pc.huber;
    float w = 1.f;
    if (fabsf(res) > huber && pc.robust) w = sqrtf(huber / fabsf(res));
    const float3 pl = cross3(q, make_float3(lx, ly, lz));
    row[0] = lx * w; row[1] = ly * w; row[2] = lz * w;
    row[3] = pl.x * w; row[4] = pl.y * w; row[5] = pl.z * w;
    row[6] = w * (-res);
    return true;
}

// The 28 products of the row's upper triangle added into the running sums, one
// fused multiply-add each (the sums are a reduction compared within a
// tolerance, not bit for bit; the rows themselves keep the reference's rounding).
// A thread adds at most 8 pixels before the warp tree and the compensated pass
// over the CTAs: the summation error stays at or below that of a
// Kahan-compensated sequential float sum without its 29 compensation registers.
__device__ __forceinline__ void accumulate(float *acc, const float row[7]) {
    int k = 0;
#pragma unroll
    for (int i = 0; i < 7; ++i)
#pragma unroll
        for (int j = i; j < 7; ++j, ++k) acc[k] = __fmaf_rn(row[i], row[j], acc[k]);
    acc[28] += 1.0f;
}

// Warp sum of 29 per-lane values by recursive halving: at each of the five
// steps a lane keeps half of its values and adds its partner's copy of them
// (xor partner), so the warp moves 31 values per lane instead of 29 x 5.  On
// return lane l (l < 29) holds the warp total of value l.  Fixed pattern:
// deterministic.
template <int N>
__device__ __forceinline__ void halve_step(float (&v)[32], int lane) {
    const bool upper = (lane & N) != 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const float send = upper ? v[i] : v[i + N];
        const float keep = upper ? v[i + N] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, N);
    }
}

__device__ __forceinline__ float warp_sum29(const float (&acc)[29]) {
    const int lane = threadIdx.x & 31;
    float v[32];
#pragma unroll
    for (int k = 0; k < 29; ++k) v[k] = acc[k];
    v[29] = v[30] = v[31] = 0.f;
    halve_step<16>(v, lane);
    halve_step<8>(v, lane);
    halve_step<4>(v, lane);
    halve_step<2>(v, lane);
    halve_step<1>(v, lane);
    return v[0];
}

constexpr int kCtaPixels = kReduceThreads * kReducePixelsPerThread;  // 1024 contiguous pixels per CTA
constexpr int kHalfThreads = kReduceThreads / 2;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// Shared memory of a reduction CTA.  The last CTA of a session reuses the
// staging tile for the sum of the partial records (sum_partials), so the sum
// costs no shared memory of its own: 8 KB more per CTA measured slower, L1
// (which the projected gathers hit 55% of the time) giving way to it.
struct ReduceSmem {
    float warp_sums[kReduceThreads / 32][29];
    __align__(16) float4 s_v[kCtaPixels];
    __align__(16) float4 s_n[kCtaPixels];
    __align__(16) float s_i[kCtaPixels];
};

// One CTA's partial sums over pixels [cta*1024, cta*1024+1024) of a level.
// The reference frame's vertices, normals and intensities of the tile (36 KB)
// are staged in shared memory with asynchronous 16-byte copies issued at once,
// so each pixel then waits for a single round trip: the gather of the current
// frame at its projection.  Warps 0-3 accumulate ICP rows, warps 4-7
// photometric rows (29 sums per thread), each thread 8 pixels 128 apart; warp
// p and warp p + 4 read the same pixels, so that pair stages them and waits at
// its own 64-thread barrier (staging the whole tile behind the CTA-wide barrier
// measured 1.4% slower over the track phase).  Warp
// shuffle tree, then a fixed-order pass over the four warps of each half.
// Writes 58 floats to part.  The caller issues the tile's copies first
// (stage_ref_tile), so that they are in flight while it loads the pose.
__device__ __forceinline__ void stage_ref_tile(ReduceSmem &sm, const SessionView &sv, int level, int rs, int cta,
                                               int tile) {
    float4 *s_v = sm.s_v, *s_n = sm.s_n;
    float *s_i = sm.s_i;
    const int P = sv.lv[level].w * sv.lv[level].h;
    const int first = cta * tile;  // tile <= kCtaPixels, a multiple of 4 (16-byte aligned copies)
    const int n = min(tile, P - first);
    {
        // Warp p (ICP rows) and warp p + 4 (photometric rows) read the same
        // pixels, c = 128 i + 32 p + lane: the pair stages those alone and meets
        // at its own 64-thread barrier instead of the CTA's.
        const int ln = threadIdx.x & 31, wd = threadIdx.x >> 5, pair = wd & 3;
        const float4 *gv = sv.vmap[rs][level] + first, *gn = sv.nmap[rs][level] + first;
        const float *gi = sv.inten[rs][level] + first;
        if (wd < 4) {  // vertices and normals
#pragma unroll
            for (int i = 0; i < kCtaPixels / kHalfThreads; ++i) {
                const int c = i * kHalfThreads + 32 * pair + ln;
                if (c < n) {
                    cp_async16(&s_v[c], gv + c);
                    cp_async16(&s_n[c], gn + c);
                }
            }
        } else {  // intensities in 16-byte chunks of 4 pixels; a chunk that would run
                  // past the image's last pixel is copied pixel by pixel instead, so
                  // nothing past the image is read
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int q = ln + 32 * j;  // 8 runs of the pair's pixels x 8 chunks
                const int c = (q >> 3) * kHalfThreads + 32 * pair + 4 * (q & 7);
                if (c + 4 <= n) {
                    cp_async16(&s_i[c], gi + c);
                } else {
                    for (int k = c; k < n; ++k) s_i[k] = gi[k];
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
}

template <bool PACKED>
__device__ __forceinline__ void cta_partial(ReduceSmem &sm, const SessionView &sv, int level, int rs, int cs,
                                            const M34 &T, float stddev, float huber, int cta, int tile, float *part) {
    auto &warp_sums = sm.warp_sums;
    float4 *s_v = sm.s_v, *s_n = sm.s_n;
    float *s_i = sm.s_i;
    const PhotoConst pc = photo_const(stddev, huber);
    const LevelIn in = level_in(sv, level, cs);
    const int P = sv.lv[level].w * sv.lv[level].h;
    const int first = cta * tile;
    const int n = min(tile, P - first);
    {
        // the pair's own copies done, then its 64-thread barrier
        const int pair = (threadIdx.x >> 5) & 3;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
    }
    const int half = threadIdx.x / kHalfThreads, t = threadIdx.x % kHalfThreads;
    float acc[29];
#pragma unroll
    for (int k = 0; k < 29; ++k) acc[k] = 0.f;
    if (n == kCtaPixels) {
        // a full tile (every CTA but a level's last): a fixed trip count with no
        // bound test lets the compiler overlap one pixel's gathers with the
        // previous pixel's rows (track phase 3.92 -> 3.72 ms against the loop below)
#pragma unroll 2
        for (int i = 0; i < kCtaPixels / kHalfThreads; ++i) {
            const int c = t + i * kHalfThreads;
            float row[7];
            const bool ok = half == 0 ? icp_row(in, T, s_v[c], s_n[c], row)
                                      : rgb_row<PACKED>(sv, level, cs, in, T, pc, s_v[c], s_i[c], row);
            if (ok) accumulate(acc, row);
        }
    } else {
#pragma unroll 2
        for (int i = 0; i < kCtaPixels / kHalfThreads; ++i) {
            const int c = t + i * kHalfThreads;
            if (c >= n) break;
            float row[7];
            const bool ok = half == 0 ? icp_row(in, T, s_v[c], s_n[c], row)
                                      : rgb_row<PACKED>(sv, level, cs, in, T, pc, s_v[c], s_i[c], row);
            if (ok) accumulate(acc, row);
        }
    }
    const float total = warp_sum29(acc);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane < 29) warp_sums[wid][lane] = total;
    __syncthreads();
    if (lane < 29 && (wid == 0 || wid == 4)) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) s += warp_sums[wid + w][lane];
        part[(wid == 0 ? 0 : 29) + lane] = s;
    }
}

// Compensated float accumulation: s + c carries the running sum, c the
// rounding errors of the additions, each found exactly by the branch-free
// TwoSum of Knuth (TAOCP vol. 2, 4.2.2) / Moller (1965).  Needs every
// operation rounded as written (no contraction, no reassociation).
struct FSum {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = s + x;
        const float bp = t - s;
        c += (s - (t - bp)) + (x - bp);
        s = t;
    }
    __device__ __forceinline__ void add(const FSum &o) {
        add(o.s);
        c += o.c;
    }
};

// Sum of the n partial records, in a fixed order, by compensated float
// addition (a single CTA adding thousands of values in FP64 is bound by this
// part's FP64 rate, ~12 us at 300 records): thread t reads the 16-byte chunk
// t % 16 (columns 4(t % 16) .. +3) of records t / 16, t / 16 + 16, ..., then the
// 16 record groups are combined in group order and widened to double.
constexpr int kSumGroups = kReduceThreads / (kPartialStride / 4);  // 16
static_assert(sizeof(float2) * kSumGroups * kPartialStride <= sizeof(float4) * kCtaPixels,
              "the group sums fit in the staging tile");
__device__ __forceinline__ void sum_partials(ReduceSmem &sm, const float *parts, int n, double *total) {
    auto grp = reinterpret_cast<float2 (*)[kPartialStride]>(sm.s_v);  // the tile is dead by now
    const int g = threadIdx.x / (kPartialStride / 4), q = threadIdx.x % (kPartialStride / 4);
    FSum s0, s1, s2, s3;
    const float4 *p4 = reinterpret_cast<const float4 *>(parts) + q;
#pragma unroll 4
    for (int c = g; c < n; c += kSumGroups) {
        const float4 v = __ldcg(p4 + (size_t)c * (kPartialStride / 4));
        s0.add(v.x);
        s1.add(v.y);
        s2.add(v.z);
        s3.add(v.w);
    }
    grp[g][4 * q] = make_float2(s0.s, s0.c);
    grp[g][4 * q + 1] = make_float2(s1.s, s1.c);
    grp[g][4 * q + 2] = make_float2(s2.s, s2.c);
    grp[g][4 * q + 3] = make_float2(s3.s, s3.c);
    __syncthreads();
    if (threadIdx.x < kReduceWidth) {
        FSum t;
#pragma unroll
        for (int h = 0; h < kSumGroups; ++h) {
            const float2 v = grp[h][threadIdx.x];
            FSum o;
            o.s = v.x;
            o.c = v.y;
            t.add(o);
        }
        total[threadIdx.x] = (double)t.s + (double)t.c;
    }
    __syncthreads();
}

struct ReduceArgs {
    int level, iter, once, defer;
    float pose[12];
    float stddev;
};

__device__ __forceinline__ void gn_epilogue(const SessionView &sv, TrackState *ts, int level, int iter, const double *s);

// Whether session `sv` runs this (level, iteration): the schedule of
// compute_transform (icp_tracker.cpp:33-50) with its early `break` per level.
__device__ __forceinline__ bool session_runs(const SessionView &sv, const ReduceArgs &a) {
    if (!sv.active || a.level >= sv.levels) return false;
    if (a.once) return true;
    const TrackState *ts = sv.ts;
    if (!ts->tracking || a.iter >= sv.max_iter[a.level]) return false;
    return !(a.iter > 0 && ts->level_done);
}

// One CTA per (tile, session): the session's sum over 1024 reference pixels
// of the ICP and photometric rows; the CTA that completes the session's last
// tile adds the partials in a fixed order and takes the Gauss-Newton step.
// Sessions that have left the level, or do not track this frame, return at
// once.
__global__ void __launch_bounds__(kReduceThreads, 4) gn_reduce_kernel(const SessionView *__restrict__ svs, ReduceArgs a) {
    const SessionView &sv = svs[blockIdx.y];
    const int level = a.level;
    if (!session_runs(sv, a) || blockIdx.x >= sv.red_ctas[level]) return;
    TrackState *ts = sv.ts;
    const int rs = ts->idx, cs = 1 - rs;
    // the reference tile's copies first: in flight while the pose is loaded
    __shared__ ReduceSmem sm;
    stage_ref_tile(sm, sv, level, rs, blockIdx.x, sv.red_tile[level]);
    __shared__ M34 T;
    __shared__ float stddev_s, huber_s;
    if (!a.once && threadIdx.x < 12) T.m[threadIdx.x] = (float)ts->est[threadIdx.x];  // one conversion, not twelve
    if (threadIdx.x == 32) {
        if (a.once) {
#pragma unroll
            for (int i = 0; i < 12; ++i) T.m[i] = a.pose[i];
        }
        stddev_s = a.once ? a.stddev : a.iter == 0 ? 0.f : ts->stddev;
        huber_s = photo_huber(stddev_s);
    }
    __syncthreads();
    cta_partial<true>(sm, sv, level, rs, cs, T, stddev_s, huber_s, blockIdx.x, sv.red_tile[level],
                sv.partials + (size_t)blockIdx.x * kPartialStride);
    if (a.defer) return;  // gn_step_kernel, launched next, sums the partials and takes the step
    __threadfence();
    __syncthreads();
    __shared__ unsigned int ticket;
    if (threadIdx.x == 0) ticket = atomicAdd(reinterpret_cast<unsigned *>(sv.ctr + C_TICKET), 1u);
    __syncthreads();
    if (ticket != (unsigned)sv.red_ctas[level] - 1u) return;
    __threadfence();
    __shared__ double total[kReduceWidth];
    sum_partials(sm, sv.partials, sv.red_ctas[level], total);
    if (threadIdx.x < kReduceWidth) ts->last_sums[threadIdx.x] = total[threadIdx.x];
    if (threadIdx.x == 0) sv.ctr[C_TICKET] = 0;
    if (!a.once && threadIdx.x < 64) gn_epilogue(sv, ts, level, a.iter, total);  // two warps
}

// The session's sum of the partial records and the Gauss-Newton step, as the
// last CTA of gn_reduce_kernel takes them, in a launch of its own (one CTA per
// session) after a deferred reduction: the reduction's CTAs then end without a
// fence and a ticket.
__global__ void __launch_bounds__(kReduceThreads) gn_step_kernel(const SessionView *__restrict__ svs, ReduceArgs a) {
    const SessionView &sv = svs[blockIdx.x];
    if (!session_runs(sv, a)) return;
    __shared__ ReduceSmem sm;
    __shared__ double total[kReduceWidth];
    sum_partials(sm, sv.partials, sv.red_ctas[a.level], total);
    if (threadIdx.x < kReduceWidth) sv.ts->last_sums[threadIdx.x] = total[threadIdx.x];
    if (threadIdx.x < 64) gn_epilogue(sv, sv.ts, a.level, a.iter, total);
}

// The bookkeeping of DenseTracking::compute_transform (icp_tracker.cpp:93-139)
// after the step of (level, iter): errors, counts and the break of the level.
// True when the step is taken back (Revertable::revert).
__device__ __forceinline__ bool gn_books(const SessionView &sv, TrackState *ts, int level, int iter, const double *s) {
    const float r_icp = (float)s[27], n_icp = (float)s[28];
    const float r_rgb = (float)s[29 + 27], n_rgb = (float)s[29 + 28];
    const float last_icp = (iter == 0) ? FLT_MAX : ts->icp_error;
    const float last_rgb = (iter == 0) ? FLT_MAX : ts->rgb_error;
    int icp_count = (iter == 0) ? 0 : ts->icp_count;
    int rgb_count = (iter == 0) ? 0 : ts->rgb_count;
    ts->iterations += 1;
    ts->level_iters[level] += 1;
    ts->pixel_iterations += (long long)sv.lv[level].w * sv.lv[level].h;
    ts->icp_inliers = n_icp;
    ts->rgb_inliers = n_rgb;
    ts->level_done = 0;
    ts->stddev = sqrtf(r_rgb / (n_rgb - 6.0f));
    float icp_error = sqrtf(r_icp) / n_icp;
    if (isnan(icp_error)) {
        ts->invalid = 1;
        ts->level_done = 1;
        ts->icp_error = icp_error;
        return false;
    }
    if (icp_error > last_icp) {
        if (icp_count >= 2) {
            ts->level_done = 1;
            return true;
        }
        icp_count++;
        icp_error = last_icp;
    } else {
        icp_count = 0;
    }
    ts->icp_error = icp_error;
    ts->icp_count = icp_count;
    float rgb_error = sqrtf(r_rgb) / n_rgb;
    if (isnan(rgb_error)) {
        ts->invalid = 1;
        ts->level_done = 1;
        ts->rgb_error = rgb_error;
        return false;
    }
    if (rgb_error > last_rgb) {
        if (rgb_count >= 2) {
            ts->level_done = 1;
            return true;
        }
        rgb_count++;
        rgb_error = last_rgb;
    } else {
        rgb_count = 0;
    }
    ts->rgb_error = rgb_error;
    ts->rgb_count = rgb_count;
    return false;
}

// Host loop body of DenseTracking::compute_transform (icp_tracker.cpp:52-139),
// run by the first two warps of a CTA: create_jtjjtr (reduce_sum.h:48-61) into
// the float matrices, A = w_icp H_icp + w_rgb H_rgb and b likewise widened to
// double, the LDL^T solve and T <- exp(xi) T on the first warp; the books on
// the second, which has the other FP32 and memory work to itself meanwhile.
__device__ __forceinline__ void gn_epilogue(const SessionView &sv, TrackState *ts, int level, int iter, const double *s) {
    const int lane = threadIdx.x & 31;
    __shared__ int revert;
    if (threadIdx.x >= 32) {
        if (lane == 0) revert = gn_books(sv, ts, level, iter, s) ? 1 : 0;
        __syncwarp();
        asm volatile("bar.sync 5, 64;" ::: "memory");
        return;
    }
    // lane p = 4 i + j < 12 holds column j of the estimate
    const int i = lane < 12 ? lane / 4 : 0, j = lane & 3;
    const double t0 = ts->est[j], t1 = ts->est[4 + j], t2 = ts->est[8 + j];
    // lane tri6(r, c) (r >= c, r < 6): A[r][c]; lane 21 + c: b[c].  The packed
    // index of (i, j), i <= j < 7, is 7 i - i (i - 1) / 2 + (j - i); b is column 6.
    const int r = tri_row(lane), c = lane < 27 ? lane - r * (r + 1) / 2 : 0;
    const int k = 7 * c - c * (c - 1) / 2 + (r - c);
    const double a = lane < 27 ? (double)(sv.w_icp * (float)s[k] + sv.w_rgb * (float)s[29 + k]) : 0.0;
    const double xi = ldlt_solve6_warp(a);
    const double next = se3_exp_mul_warp(xi, t0, t1, t2);
    asm volatile("bar.sync 5, 64;" ::: "memory");
    if (lane < 12) {
        const double old = i == 0 ? t0 : i == 1 ? t1 : t2;
        ts->est_prev[lane] = old;
        ts->est[lane] = revert ? old : next;
    }
}

// frame_mode 1: System frame (track only when a reference exists); 0: gbf_track.
__device__ __forceinline__ void track_begin(TrackState *ts, int frame_mode) {
    ts->tracking = frame_mode ? ts->has_ref : 1;
    // Revertable(initial_estimate): curr = init, prev = identity
    pose_copy(ts->init, ts->est);
    pose_identity(ts->est_prev);
    ts->invalid = 0;
    ts->iterations = 0;
    for (int l = 0; l < kMaxLevels; ++l) ts->level_iters[l] = 0;
    ts->level_done = 0;
    ts->icp_error = FLT_MAX;
    ts->rgb_error = FLT_MAX;
    ts->stddev = 0.f;
    ts->icp_count = ts->rgb_count = 0;
}

// The success test of the tracking result (icp_tracker.cpp:145), |log(est^-1 init)| <= 0.1.
__device__ __noinline__ bool moved_too_far(const double *est, const double *init) {
    double inv[12], rel[12];
    pose_inverse(est, inv);
    pose_mul(inv, init, rel);
    return !(se3_log_norm(rel) <= 0.1);
}

// The same test decided in FP32 where the norm is clearly on one side: -1 when it
// is not (near the bound, large rotations or coordinates, non-finite poses).  With
// |elements| <= 50 and a rotation below 0.46 rad (trace > 2.8) every step is
// within a few 1e-6 of the FP64 one, against a margin of 1e-3.
__device__ __forceinline__ int moved_too_far_f32(const float *e, const float *init) {
    float m = 0.f;
    bool finite = true;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        m = fmaxf(m, fmaxf(fabsf(e[i]), fabsf(init[i])));
        finite = finite && isfinite(e[i]) && isfinite(init[i]);
    }
    float R[9], t[3], d[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) d[k] = init[k * 4 + 3] - e[k * 4 + 3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        t[i] = e[i] * d[0] + e[4 + i] * d[1] + e[8 + i] * d[2];
#pragma unroll
        for (int j = 0; j < 3; ++j) R[i * 3 + j] = e[i] * init[j] + e[4 + i] * init[4 + j] + e[8 + i] * init[8 + j];
    }
    if (!finite || !(m <= 50.f) || !(R[0] + R[4] + R[8] > 2.8f)) return -1;
    float wx = 0.5f * (R[7] - R[5]), wy = 0.5f * (R[2] - R[6]), wz = 0.5f * (R[3] - R[1]);
    const float s = norm3(wx, wy, wz);
    const float k = s > 1e-4f ? asinf(fminf(s, 1.f)) / s : 1.f;
    wx *= k;
    wy *= k;
    wz *= k;
    const float th2 = wx * wx + wy * wy + wz * wz;
    // rho = t - w x t / 2 + f w x (w x t), f = 1/12 + th^2/720 + ...
    const float3 w = make_float3(wx, wy, wz), tv = make_float3(t[0], t[1], t[2]);
    const float3 c1 = cross3(w, tv), c2 = cross3(w, c1);
    const float f = 1.f / 12.f + th2 * (1.f / 720.f + th2 * (1.f / 30240.f));
    const float rx = tv.x - 0.5f * c1.x + f * c2.x, ry = tv.y - 0.5f * c1.y + f * c2.y, rz = tv.z - 0.5f * c1.z + f * c2.z;
    const float n = sqrtf(rx * rx + ry * ry + rz * rz + th2);
    return n < 0.099f ? 0 : n > 0.101f ? 1 : -1;
}

// Tracking result (icp_tracker.cpp:143-155), by one warp (all lanes); frame_mode 1
// also applies the System / DenseOdometry bookkeeping (rgbd_odometry.cpp:39-41): pose update
// and reference swap.  The pose products take one lane per element; with one
// thread, and the FP64 logarithm of every frame's motion, this took 18 us.
__device__ __forceinline__ void track_finish(const SessionView &sv, TrackState *ts, int frame_mode) {
    const int lane = threadIdx.x & 31, p = lane < 12 ? lane : 0;
    const double identity = (p == 0 || p == 5 || p == 10) ? 1.0 : 0.0;
    const bool tracking = ts->tracking;
    double pose = ts->pose[p], update = ts->update[p], init = ts->init[p];
    bool success = ts->success;
    if (tracking) {
        const double est = ts->est[p];
        float e[12], f[12];
#pragma unroll
        for (int i = 0; i < 12; ++i) {
            e[i] = __shfl_sync(0xffffffffu, (float)est, i);
            f[i] = __shfl_sync(0xffffffffu, (float)init, i);
        }
        int far = moved_too_far_f32(e, f);
        if (far < 0) {
            if (lane == 0) far = moved_too_far(ts->est, ts->init) ? 1 : 0;
            far = __shfl_sync(0xffffffffu, far, 0);
        }
        const bool finite = __all_sync(0xffffffffu, isfinite(est));
        success = !(ts->invalid || far || !finite);
        update = pose_inverse_warp(est);
        if (!success) update = identity;
        if (frame_mode) pose = pose_mul_warp(pose, update);
        if (lane == 0) {
            if (!finite) raise_flag(sv, GBF_FLAG_NAN_POSE);
            if (!success && frame_mode) raise_flag(sv, GBF_FLAG_TRACK_FAILED);
        }
    } else if (frame_mode) {
        success = true;
        update = identity;
    }
    const double inv = pose_inverse_warp(frame_mode ? pose : update);
    if (frame_mode) {
        // the next frame's initial estimate: no motion (the reference), or
        // with the constant-velocity prior the motion this frame tracked
        init = identity;
        if (sv.motion_prior && tracking && success) init = pose_inverse_warp(update);
    }
    __syncwarp();
    if (lane < 12) {
        if (tracking || frame_mode) ts->update[p] = update;
        if (frame_mode) {
            ts->pose[p] = pose;
            ts->init[p] = init;
            ts->map_pose[p] = pose;
            ts->map_twc[p] = (float)pose;  // update_map_floats
            ts->map_tcw[p] = (float)inv;
        }
    }
    if (lane == 0) {
        if (tracking || frame_mode) ts->success = success ? 1 : 0;
        if (frame_mode) {
            ts->idx = 1 - ts->idx;
            ts->has_ref = 1;
            ts->frame_index += 1;
        }
    }
    __syncwarp();
}

__global__ void track_begin_kernel(const SessionView *__restrict__ svs, int frame_mode) {
    const SessionView &sv = svs[blockIdx.x];
    if (!sv.active || threadIdx.x != 0) return;
    track_begin(sv.ts, frame_mode);
    sv.ctr[C_TICKET] = 0;
}

__global__ void track_finish_kernel(const SessionView *__restrict__ svs, int frame_mode) {
    const SessionView &sv = svs[blockIdx.x];
    if (sv.active) track_finish(sv, sv.ts, frame_mode);
}

// ---------------------------------------------------------------------------
// A whole tracking run (every level and iteration, from the initial estimate to
// the frame's pose) in one launch, for launches of few sessions.
//
// What bounds such a run is latency.  A launch per iteration costs one 640x480
// session about 18 us: the launch, the dependent loads from the descriptor to the
// first pixel, four rounds of gathers one after another, a last CTA that sums
// the records and the step, of which the chip is busy for a quarter.  Here one
// CTA per SM stays for the run, its code and the maps it gathers from in its
// caches.  512 threads make the two rows of two pixels each of a 1024-pixel tile,
// every gather of the tile in flight at once, into shared memory (zeros for a
// rejected row); then half of the threads sum the 29 products of an eight-pixel chain
// each, where holding 29 sums while gathering leaves registers for two pixels in
// flight (all threads, two to a chain with half of the products each, read the rows
// twice and took 3% longer over a 1280x720 frame's run: the rows' way through shared
// memory weighs as much as the arithmetic).  CTA 0 makes no rows: it sums the tiles'
// records as they arrive, takes the step on the tracking state in its shared memory and
// publishes the next pose, so that the step's code stays in one SM's instruction cache.
// An iteration then takes 9 us at 320x240 and below, 13 at 640x480 and 24 at 1280x720
// (one, two and six tiles per CTA of 2.4 us each: 1.5 the rows, 0.65 the chains; the step
// 3.7; each hop between CTAs 0.7; the records 1 to 2), the run of a 640x480 frame 0.25
// -> 0.15 ms.  1024 threads of 64 registers spilled (0.25 ms);
// the step by whichever CTA came last ran 25% slower from cold instruction
// caches; coarse tiles split over two or four CTAs cost more in records than they saved.
//
// Every sum keeps the terms and the order of gn_reduce_kernel: a chain adds
// pixels t, t + 128, ... of the tile in turn (fused multiply-adds; a zero row
// adds nothing), a warp adds its 32 chains in a butterfly (xor 16, 8, 4, 2, 1),
// the tile adds its four warps in order, the records follow as in sum_partials.
constexpr int kTrackThreads = 512;
constexpr int kTrackPixels = kCtaPixels / kTrackThreads;  // of a tile per thread
struct TrackSmem {
    float4 lo[2][kCtaPixels];  // ICP, photometric: row[0..3]
    float4 hi[2][kCtaPixels];  // row[4..6], 1 for a valid row
    float warp_sums[4][kReduceWidth];
    float2 grp[kSumGroups][kReduceWidth];
    double total[kReduceWidth];
    TrackState ts;  // CTA 0: the run's tracking state
    float pose[12];
    float stddev, huber;
    unsigned seen, base, order;
    int item, lost, crew;
};

// icp_row and rgb_row of one pixel, with their gathers issued together (a row
// rejected before its gather reads pixel 0 and is masked after).
__device__ __forceinline__ void pixel_rows(const LevelIn &K, const M34 &T, const PhotoConst &pc, const float4 pt,
                                           const float4 nr, float il, float4 *icp_lo, float4 *icp_hi, float4 *rgb_lo,
                                           float4 *rgb_hi) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float3 p = T.apply(pt.x, pt.y, pt.z);
    const float zi = __frcp_rn(p.z);
    const int u = __float2int_rd(((p.x * zi) * K.fx + K.cx) + 0.5f);
    const int w = __float2int_rd(((p.y * zi) * K.fy + K.cy) + 0.5f);
    bool ok = !isnan(pt.x) && !(u < 0 || w < 0 || u >= K.w || w >= K.h);
    const int q = ok ? w * K.w + u : 0;
    // p.x / p.z and p.y / p.z from the reciprocal at hand (div_rn_by; where z has none,
    // the quotient is outside the image or NaN either way)
    const float u0 = div_rn_by(p.x, p.z, zi) * K.fx + K.cx;
    const float v0 = div_rn_by(p.y, p.z, zi) * K.fy + K.cy;
    bool okr = !(pt.w < 0 || isnan(pt.x)) && isfinite(il) &&
               (u0 >= 2 && u0 < (float)(K.w - 2) && v0 >= 2 && v0 < (float)(K.h - 2));
    const int iu = (int)floorf(u0), iv = (int)floorf(v0);
    const float4 *r0 = K.igd + (okr ? iv * K.w + iu : 0);
    const float4 vc = K.vcur[q], nc = K.ncur[q];
    const float4 a = r0[0], b = r0[1], c = r0[K.w], d = r0[K.w + 1];
    {
        const float3 ng = T.rotate(nr.x, nr.y, nr.z);
        const float dist2 = norm3_sq(p.x - vc.x, p.y - vc.y, p.z - vc.z);
        const float3 cr = cross3(make_float3(nc.x, nc.y, nc.z), ng);
        const float sine2 = norm3_sq(cr.x, cr.y, cr.z);
        ok = ok && sine2 < K.angle2 && dist2 <= K.dist2 && !isnan(nc.x) && !isnan(ng.x);
        const float3 x = cross3(p, ng);
        const float r = dot3(ng, make_float3(vc.x - p.x, vc.y - p.y, vc.z - p.z));
        *icp_lo = ok ? make_float4(ng.x, ng.y, ng.z, x.x) : zero;
        *icp_hi = ok ? make_float4(x.y, x.z, r, 1.f) : zero;
    }
    {
        const float ax = u0 - (float)iu, ay = v0 - (float)iv, bx = 1.0f - ax, by = 1.0f - ay;
        const float ic = (a.x * bx + b.x * ax) * by + (c.x * bx + d.x * ax) * ay;
        const float dx = (a.y * bx + b.y * ax) * by + (c.y * bx + d.y * ax) * ay;
        const float dy = (a.z * bx + b.z * ax) * by + (c.z * bx + d.z * ax) * ay;
        okr = okr && (dx > 2 || dy > 2) && isfinite(ic) && isfinite(dx) && isfinite(dy);
        const float lx = (dx * K.fx) * zi, ly = (dy * K.fy) * zi;
        const float lz = (-(lx * p.x + ly * p.y)) * zi;
        float res = ic - il;
        if (pc.normalise) res = div_rn_by(res, pc.div, pc.inv);
        float wt = 1.f;
        if (fabsf(res) > pc.huber && pc.robust) wt = sqrtf(pc.huber / fabsf(res));
        const float3 x = cross3(p, make_float3(lx, ly, lz));
        *rgb_lo = okr ? make_float4(lx * wt, ly * wt, lz * wt, x.x * wt) : zero;
        *rgb_hi = okr ? make_float4(x.y * wt, x.z * wt, wt * (-res), 1.f) : zero;
    }
}

// The 29 sums of chain t's eight rows (t, t + 128, ... of the tile).
__device__ __forceinline__ void chain_sums(const float4 *lo, const float4 *hi, int t, float (&acc)[29]) {
#pragma unroll
    for (int k = 0; k < 29; ++k) acc[k] = 0.f;
#pragma unroll
    for (int i = 0; i < kCtaPixels / kHalfThreads; ++i) {
        const float4 a = lo[t + i * kHalfThreads], b = hi[t + i * kHalfThreads];
        const float row[7] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z};
        const float count = acc[28] + b.w;  // a rejected pixel's row is all zeros
        accumulate(acc, row);
        acc[28] = count;
    }
}

// A CTA of the run waits for another at most this long (CTA 0: SessionView::track_wait_ns).
// The CTAs of a run are resident (gather_crew) and a step takes microseconds: the limit
// only bounds a wait that cannot happen.
struct WaitLimit {
    long long ns, t0 = 0;
    int n = 0, every;
    bool ran_out = false;
    __device__ __forceinline__ explicit WaitLimit(long long limit) : ns(limit), every(limit > 0 ? 63 : 0) {}
    __device__ __forceinline__ bool over() {
        if (++n & every) return false;
        long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (!t0) t0 = t;
        return ran_out = t - t0 >= ns;
    }
};

__device__ __forceinline__ unsigned ld_acquire(const int *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned atom_add(int *p, unsigned n) {
    unsigned v;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "r"(n) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// What one CTA of a run hands to another travels as 8-byte words of (value,
// sequence number): a word that carries its own number needs no fence and no
// second round trip, and leaves the readers' L1, with the maps they gather from,
// alone.  CTA 0 publishes 14 of them after each step -- the estimate's 12 floats, the
// photometric deviation and the work item; the others write the sums of their
// tile, numbered like the publication that will follow.  The numbers run on over the
// session's runs and wrap: one is newer by the sign of the difference.
constexpr int kPubWords = 14;
constexpr unsigned kRunClosed = 1u << 20;  // above any count of CTAs
__device__ __forceinline__ unsigned long long tagged(unsigned number, unsigned value) {
    return ((unsigned long long)number << 32) | value;
}
__device__ __forceinline__ unsigned number_of(unsigned long long word) { return (unsigned)(word >> 32); }

// A run's work items are (level, iteration) packed; 0 is its end.
__device__ __forceinline__ int first_item(const SessionView &sv, int level) {
    while (level >= 0 && sv.max_iter[level] == 0) --level;
    return (level + 1) << 10;
}

// One tile's sums: word q of record `rec`.
__device__ __forceinline__ unsigned long long *record_word(const SessionView &sv, int rec, int q) {
    return sv.track_rec + (size_t)rec * kPartialStride + q;
}

// The sums of the item numbered `number`, by all threads of CTA 0: warp g waits
// for ten of the records g, g + 16, ... at a time (a lane per record looks at its first
// word), then lane q adds columns 2 q and 2 q + 1 of them in turn; the 16 groups follow in
// order (the sums and the order of sum_partials).  The words are read twenty in
// flight and checked by their numbers: one relaxed load a word, since another CTA may be
// storing it (a plain load of two words promises neither whole words nor that a
// store is seen, and took longer: a 1280x720 run 224 us, 217 so).  Only the records that come last are
// then left to read when the last tile is done (waiting for thirty at a time, as many as fit
// the lanes, left a 1280x720 image's whole second half).  Records past the last
// count as zeros, which add nothing.
static_assert(kTrackThreads == 32 * kSumGroups, "a warp per record group");
__device__ __forceinline__ bool sum_records(TrackSmem &sm, const SessionView &sv, int n, unsigned number) {
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31, q = min(2 * lane, kReduceWidth - 2);
    WaitLimit limit(sv.track_wait_ns);
    FSum s0, s1;
    constexpr int kBatch = 10;  // at most a record per lane
    for (int c = g; c < n; c += kBatch * kSumGroups) {
        const int r = c + lane * kSumGroups;
        const bool mine = lane < kBatch && r < n;
        while (!__all_sync(0xffffffffu, !mine || number_of(ld_relaxed(record_word(sv, r, 0))) == number) &&
               !__any_sync(0xffffffffu, limit.over())) {}
        ulonglong2 w[kBatch];
        bool all;
        do {
            all = true;
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                w[i] = make_ulonglong2(tagged(number, 0u), tagged(number, 0u));
                const unsigned long long *p = record_word(sv, c + i * kSumGroups, q);
                if (c + i * kSumGroups < n) w[i] = make_ulonglong2(ld_relaxed(p), ld_relaxed(p + 1));
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) all = all && number_of(w[i].x) == number && number_of(w[i].y) == number;
        } while (!__all_sync(0xffffffffu, all) && !__any_sync(0xffffffffu, limit.over()));
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            s0.add(__uint_as_float((unsigned)w[i].x));
            s1.add(__uint_as_float((unsigned)w[i].y));
        }
    }
    sm.grp[g][q] = make_float2(s0.s, s0.c);
    sm.grp[g][q + 1] = make_float2(s1.s, s1.c);
    const bool ok = __syncthreads_and(!limit.ran_out);
    if (threadIdx.x < kReduceWidth) {
        FSum t;
#pragma unroll 4
        for (int h = 0; h < kSumGroups; ++h) {
            const float2 v = sm.grp[h][threadIdx.x];
            FSum o;
            o.s = v.x;
            o.c = v.y;
            t.add(o);
        }
        sm.total[threadIdx.x] = (double)t.s + (double)t.c;
    }
    __syncthreads();
    return ok;
}

// The newest publication after number `seen`, by one warp: lanes < 14 get the
// values.  False when the wait ran out.
__device__ __forceinline__ bool read_pub(const unsigned long long *pub, unsigned &seen, unsigned &value) {
    const int lane = threadIdx.x & 31;
    WaitLimit limit(kTrackWaitNs);
    for (;;) {
        const unsigned long long w = lane < kPubWords ? ld_relaxed(pub + lane) : 0ull;
        const unsigned n = number_of(w), n0 = __shfl_sync(0xffffffffu, n, 0);
        if (__all_sync(0xffffffffu, lane >= kPubWords || n == n0) && (int)(n0 - seen) > 0) {
            seen = n0;
            value = (unsigned)w;
            return true;
        }
        if (__any_sync(0xffffffffu, lane == 0 && limit.over())) return false;
    }
}

// The steps of a run: CTA 0 adds each item's records, takes the step on the
// tracking state in shared memory and publishes what follows.
__device__ __forceinline__ void track_steps(TrackSmem &sm, const SessionView &sv, int item, unsigned seen, bool lost,
                                            int frame_mode) {
    TrackState *ts = &sm.ts;
    const int tid = threadIdx.x, lane = tid & 31;
    unsigned long long *pub = reinterpret_cast<unsigned long long *>(sv.ctr + C_TRACK_PUB);
    while (item > 0 && !lost) {
        const int level = (item >> 10) - 1, iter = item & 1023;
        lost = !sum_records(sm, sv, sv.red_ctas[level], ++seen);
        if (lost) break;
        if (tid >= 64 && tid < 64 + kReduceWidth) ts->last_sums[tid - 64] = sm.total[tid - 64];
        if (tid < 64) gn_epilogue(sv, ts, level, iter, sm.total);
        __syncthreads();
        item = ts->level_done || iter + 1 >= sv.max_iter[level] ? first_item(sv, level - 1) : item + 1;
        if (tid < kPubWords) {
            const float dev = level == (item >> 10) - 1 ? ts->stddev : 0.f;  // each level starts without one
            const float x = lane < 12 ? (float)ts->est[lane] : dev;
            st_relaxed(pub + lane, tagged(seen, lane < 13 ? __float_as_uint(x) : (unsigned)item));
        }
        __syncwarp();
    }
    __syncthreads();
    if (tid < 32) {
        if (lost) {
            // a wait ran out: the frame counts as not tracked, the other CTAs end, and the
            // numbers go on behind that of the records that may still come
            ts->invalid = 1;
            if (lane == 0) raise_flag(sv, GBF_FLAG_TRACK_WAIT);
            if (lane < kPubWords) st_relaxed(pub + lane, tagged(seen + 1, 0u));
        }
        __syncwarp();
        track_finish(sv, ts, frame_mode);
    }
    __syncthreads();
    for (int i = tid; i < (int)(sizeof(TrackState) / 4); i += kTrackThreads)
        reinterpret_cast<int *>(sv.ts)[i] = reinterpret_cast<const int *>(ts)[i];
}

// How many CTAs share a run's tiles: CTA 0 waits until the launch's ctas have arrived, or
// for so long that the rest are not about to (another stream's kernel holds their SMs,
// or the stream has fewer), and goes on with those that have: they run, and so every
// wait of the run ends, without a cooperative launch, which starts only once all can.  (A
// 320x240 frame beside a kernel of one CTA and 5 ms on another stream took 4.96 ms so,
// and takes 0.31; on a stream of 64 SMs, which refuses the cooperative grid, 0.42 ms with
// launches per iteration and 0.33 so.)  Not long where most have come, longer where few
// have, as while another kernel's CTAs end: patience of 100 or 250 us gained nothing
// beside matrix products or a batch's ticks, and cost a stream of 64 SMs 57 or 203 us.
// False when it took too long or no other CTA came.
constexpr long long kCrewQuiet = 40000, kCrewPatience = 80000;  // cycles: 20 and 40 us
__device__ __forceinline__ unsigned long long *crew_word(const SessionView &sv) {
    return reinterpret_cast<unsigned long long *>(sv.ctr + C_TRACK_CREW);
}
__device__ __forceinline__ bool gather_crew(const SessionView &sv, unsigned base, unsigned ctas, int item, unsigned seen) {
    WaitLimit limit(sv.track_wait_ns);
    const long long start = clock64();
    long long quiet = start;
    unsigned n, last = 0;
    while ((n = ld_acquire(sv.ctr + C_TRACK_ARRIVED) - base) != ctas && !limit.over()) {
        const long long t = clock64();
        if (n != last) quiet = t;
        last = n;
        if (n > 1 && t - quiet > kCrewQuiet && (2 * n > ctas || t - start > kCrewPatience)) break;
    }
    unsigned next = base + ctas;
    if (n != ctas) {
        n = atom_add(sv.ctr + C_TRACK_ARRIVED, kRunClosed) - base;
        next += kRunClosed;
    }
    sv.ctr[C_TRACK_BASE] = (int)next;
    // (a run without items publishes nothing, so that the next one starts from the same number)
    if (item > 0) st_relaxed(crew_word(sv), tagged(seen + 1, n - 1));
    return !limit.ran_out && n > 1;
}

// The tiles of a run: CTA cta of those that follow CTA 0 makes its tiles' records of each item.
__device__ __forceinline__ void track_tiles(TrackSmem &sm, const SessionView &sv, int item, unsigned seen, int rs,
                                            int cta) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned long long *pub = reinterpret_cast<const unsigned long long *>(sv.ctr + C_TRACK_PUB);
    const float qnan = __int_as_float(0x7fffffff);
    const float4 nan4 = make_float4(qnan, qnan, qnan, -1.f);
    float4 v[kTrackPixels], m[kTrackPixels];  // this thread's reference pixels of the CTA's next tile
    float il[kTrackPixels];
    int loaded = -1;  // the level they belong to
    int ctas = 0;     // not known before the first tile's rows are made
    const auto read_crew = [&]() {
        if (warp == 0) {
            WaitLimit limit(kTrackWaitNs);
            unsigned long long w = ld_relaxed(crew_word(sv));
            while (number_of(w) != seen + 1 && !limit.over()) w = ld_relaxed(crew_word(sv));
            if (lane == 0) sm.crew = limit.ran_out ? 0 : (int)(unsigned)w;
            __syncwarp();
        }
        __syncthreads();
        ctas = sm.crew;
    };
    while (item > 0) {
        const int level = (item >> 10) - 1;
        const LevelIn in = level_in(sv, level, 1 - rs);
        const int tiles = sv.red_ctas[level], P = in.w * in.h;
        const float4 *gv = sv.vmap[rs][level], *gn = sv.nmap[rs][level];
        const float *gi = sv.inten[rs][level];
        const auto load = [&](int tile) {
#pragma unroll
            for (int j = 0; j < kTrackPixels; ++j) {
                const int c = tile * kCtaPixels + tid + j * kTrackThreads;
                v[j] = m[j] = nan4;
                il[j] = qnan;
                if (c < P) {
                    v[j] = gv[c];
                    m[j] = gn[c];
                    il[j] = gi[c];
                }
            }
        };
        if (cta < tiles) {
            if (loaded != level) load(cta);
            loaded = level;
            M34 T;
#pragma unroll
            for (int i = 0; i < 12; ++i) T.m[i] = sm.pose[i];
            const PhotoConst pc = photo_const(sm.stddev, sm.huber);
            for (int tile = cta; tile < tiles; tile += ctas) {  // (ctas is known from the first one's on)
#pragma unroll
                for (int j = 0; j < kTrackPixels; ++j) {
                    const int k = tid + j * kTrackThreads;
                    pixel_rows(in, T, pc, v[j], m[j], il[j], sm.lo[0] + k, sm.hi[0] + k, sm.lo[1] + k, sm.hi[1] + k);
                }
                if (!ctas) read_crew();
                if (!ctas) return;
                // meanwhile the next tile's pixels, or the first one's again for the next iteration
                load(tile + ctas < tiles ? tile + ctas : cta);
                __syncwarp();
                __syncthreads();
                if (warp < 8) {  // ICP chains, then photometric ones
                    const int half = warp >> 2, cw = warp & 3;
                    float acc[29];
                    chain_sums(sm.lo[half], sm.hi[half], 32 * cw + lane, acc);
                    const float s = warp_sum29(acc);
                    if (lane < 29) sm.warp_sums[cw][half * 29 + lane] = s;
                }
                __syncwarp();
                __syncthreads();
                if (tid < kReduceWidth) {
                    float s = 0.f;
#pragma unroll
                    for (int w = 0; w < 4; ++w) s += sm.warp_sums[w][tid];
                    st_relaxed(record_word(sv, tile, tid), tagged(seen + 1, __float_as_uint(s)));
                }
            }
        } else {
            __syncthreads();  // every warp has the item before the next one takes its place
            if (!ctas) read_crew();
            if (!ctas) return;
        }
        if (warp == 0) {
            unsigned value = 0;
            const bool ok = read_pub(pub, seen, value);
            if (lane < 12) sm.pose[lane] = __uint_as_float(value);
            if (lane == 12) {
                sm.stddev = __uint_as_float(value);
                sm.huber = photo_huber(sm.stddev);
            }
            if (lane == 13) {
                sm.item = ok ? (int)value : -1;
                sm.seen = seen;
            }
            __syncwarp();
        }
        __syncthreads();
        item = sm.item;
        seen = sm.seen;
    }
}

__global__ void __launch_bounds__(kTrackThreads, 1)
    gn_track_kernel(const SessionView *__restrict__ svs, int frame_mode) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char track_smem[];
    TrackSmem &sm = *reinterpret_cast<TrackSmem *>(track_smem);
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active) return;
    const int tid = threadIdx.x;
    // Every CTA reads these before it arrives: what CTA 0 publishes, and the frame's
    // end, change them.
    const int rs = sv.ts->idx;
    const unsigned seen = number_of(ld_relaxed(reinterpret_cast<const unsigned long long *>(sv.ctr + C_TRACK_PUB)));
    const int item = frame_mode && !sv.ts->has_ref ? 0 : first_item(sv, sv.levels - 1);
    if (tid < 12) sm.pose[tid] = (float)sv.ts->init[tid];
    if (tid == 12) sm.stddev = sm.huber = 0.f;
    __syncwarp();
    __syncthreads();
    // The order of arrival is the CTA's place in the run, 0 that of "CTA 0" above.  Arrivals are
    // counted over the session's runs: all of a run's have been made when the next one starts.
    // A run that goes on without some of its CTAs has added kRunClosed to the count, and
    // whichever base these read, their order is past any place.
    if (tid == 0) {
        const unsigned base = ld_acquire(sv.ctr + C_TRACK_BASE);
        sm.base = base;
        sm.order = atom_add(sv.ctr + C_TRACK_ARRIVED, 1u) - base;
    }
    __syncwarp();
    __syncthreads();
    const unsigned order = sm.order, ctas = gridDim.x;
    if (order >= ctas) return;
    if (order > 0) {
        track_tiles(sm, sv, item, seen, rs, (int)order - 1);
        return;
    }
    for (int i = tid; i < (int)(sizeof(TrackState) / 4); i += kTrackThreads)
        reinterpret_cast<int *>(&sm.ts)[i] = reinterpret_cast<const int *>(sv.ts)[i];
    __syncwarp();
    __syncthreads();
    if (tid == 0) {
        track_begin(&sm.ts, frame_mode);
        sm.lost = !gather_crew(sv, sm.base, ctas, item, seen);
    }
    __syncwarp();
    __syncthreads();
    track_steps(sm, sv, item, seen, sm.lost, frame_mode);
}

}  // namespace

// Sessions whose Gauss-Newton iterations run back to back before the next
// subgroup's: a subgroup's level-0 images (about 25 MB per 640x480 session)
// then stay in L2 from one iteration to the next.
constexpr int kTrackSubgroup = 64;

// Sessions per launch from which the Gauss-Newton step runs as a launch of its
// own (gn_step_kernel) instead of in the last CTA of the reduction: with many
// sessions the reduction's CTAs then end without a fence and a ticket (two
// groups of 32 sessions: track 3.71 -> 3.46 ms, tick 10.85 -> 10.80 ms; of 64:
// 5,950 -> 6,057 frames/s); with fewer, the extra launch per iteration costs
// more than it saves (two groups of 16: 5,764 -> 5,702 frames/s; one session:
// 1,236 -> 1,165 frames/s).
constexpr int kDeferStepSessions = 32;
static bool defer_step(int sessions) { return sessions >= kDeferStepSessions; }

// Whether a launch that may take the chip tracks in one run: track 0.25 -> 0.154 ms for one 640x480 session, 0.28 -> 0.18 for
// two, 0.34 -> 0.23 for three, 0.39 -> 0.29 for four.  More sessions share the CTAs, which
// are then busy with their tiles most of the time; small images leave the run ahead of
// two concurrent groups of launches (ticks of 6 sessions at 320x240, 450 level-0 tiles, 0.80
// -> 0.76 ms; 12, 900 tiles, 1.14 -> 1.11; 16 at 256x192, 768 tiles, 1.39 -> 1.34), larger
// ones do not (8 at 448x336, 1176 tiles, 1.02 both; 16 at 320x240, 1200 tiles, 1.42 -> 1.47;
// 5 at 896x672, 2940 tiles, 1.50 -> 1.55).
constexpr int kTrackRunFew = 4, kTrackRunSessions = 16, kTrackRunTiles = 1000;
bool track_run_fits(int nslots, const Extent &ex) {
    return nslots <= kTrackRunFew || (nslots <= kTrackRunSessions && nslots * ex.max_red[0] <= kTrackRunTiles);
}

// CTAs of one launch of gn_track_kernel on the current device (one per SM), or 0 where
// it cannot be launched.
static int track_run_ctas() {
    static std::atomic<int> known[64];  // per device: CTAs + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::atomic<int> &k = known[dev & 63];
    int c = k.load(std::memory_order_acquire);
    if (c == 0) {
        int sms = 0, per = 0;
        c = 1;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            cudaFuncSetAttribute(gn_track_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(TrackSmem)) ==
                cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, gn_track_kernel, kTrackThreads, sizeof(TrackSmem)) ==
                cudaSuccess)
            c = sms * per + 1;
        k.store(c, std::memory_order_release);
    }
    return c - 1;
}

static bool takes_run(int nslots, const Extent &ex, bool alone) {
    return alone && track_run_fits(nslots, ex) && track_run_ctas() >= 2 * nslots;
}

int track_launches(int nslots, const Extent &ex, bool alone) {
    if (takes_run(nslots, ex, alone)) return 1;
    int it = 0;
    for (int l = 0; l < ex.levels; ++l) it += ex.max_iter[l];
    int n = 0;
    for (int s0 = 0; s0 < nslots; s0 += kTrackSubgroup)
        n += it * (defer_step(min(kTrackSubgroup, nslots - s0)) ? 2 : 1);
    return 2 + n;
}

void prepare_track() { track_run_ctas(); }

void launch_track(const SessionView *d_sv, int nslots, const Extent &ex, int frame_mode, bool alone, cudaStream_t st) {
    if (takes_run(nslots, ex, alone)) {
        // Not chained: its CTAs, a whole SM each, would wait in places that the level maps'
        // could use (640x480 frames, each pose read back, 366 us chained, 361 so; one after the
        // other the same).
        gn_track_kernel<<<dim3(track_run_ctas() / nslots, nslots), kTrackThreads, sizeof(TrackSmem), st>>>(d_sv,
                                                                                                          frame_mode);
        return;
    }
    track_begin_kernel<<<nslots, 32, 0, st>>>(d_sv, frame_mode);
    ReduceArgs a{};
    a.once = 0;
    for (int s0 = 0; s0 < nslots; s0 += kTrackSubgroup) {
        const int n = min(kTrackSubgroup, nslots - s0);
        for (int level = ex.levels - 1; level >= 0; --level) {
            for (int iter = 0; iter < ex.max_iter[level]; ++iter) {
                a.level = level;
                a.iter = iter;
                a.defer = defer_step(n) ? 1 : 0;
                gn_reduce_kernel<<<dim3(ex.max_red[level], n), kReduceThreads, 0, st>>>(d_sv + s0, a);
                if (a.defer) gn_step_kernel<<<n, kReduceThreads, 0, st>>>(d_sv + s0, a);
            }
        }
    }
    track_finish_kernel<<<nslots, 32, 0, st>>>(d_sv, frame_mode);
}

void launch_reduce_once(const SessionView *d_sv, const Extent &ex, int level, const float *pose12, float stddev,
                        cudaStream_t st) {
    ReduceArgs a{};
    a.once = 1;
    a.level = level;
    a.iter = 0;
    for (int i = 0; i < 12; ++i) a.pose[i] = pose12[i];
    a.stddev = stddev;
    gn_reduce_kernel<<<dim3(ex.max_red[level], 1), kReduceThreads, 0, st>>>(d_sv, a);
}

void launch_frame_finish(const SessionView *d_sv, int nslots, cudaStream_t st) {
    track_finish_kernel<<<nslots, 32, 0, st>>>(d_sv, 1);
}

namespace {
__global__ void slot_results_kernel(const SessionView *__restrict__ svs, int n, gbf_slot_result *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const SessionView &sv = svs[i];
    if (sv.tick_done) *static_cast<volatile unsigned *>(sv.tick_done) = sv.tick_number;
    gbf_slot_result r;
    if (!sv.ts) {  // empty slot
        for (int j = 0; j < 16; ++j) r.pose[j] = 0.0;
        r.tracked = 0;
        r.status = 0u;
        r.frame_index = 0;
    } else {
        const TrackState *ts = sv.ts;
        for (int j = 0; j < 12; ++j) r.pose[j] = ts->pose[j];
        r.pose[12] = r.pose[13] = r.pose[14] = 0.0;
        r.pose[15] = 1.0;
        r.tracked = ts->success;
        r.status = (uint32_t)sv.ctr[C_STATUS];
        r.frame_index = ts->frame_index;
    }
    out[i] = r;
}
}  // namespace

void launch_slot_results(const SessionView *d_sv, int nslots, gbf_slot_result *out, cudaStream_t st) {
    slot_results_kernel<<<(nslots + 127) / 128, 128, 0, st>>>(d_sv, nslots, out);
}

}  // namespace gbf

// ============================================================================
// Allocation-free ICP + photometric reduction.
//
// Some callers cannot allocate device memory at all: real-time camera loops
// that forbid allocation once they run (a cudaMalloc can block for
// milliseconds and synchronise the device), and host frameworks that hand out
// every byte of device memory through their own allocator, so that a library
// allocating behind their back would fail or break their accounting.  For them this entry
// point reduces one pyramid level of caller-owned images with no session and no
// cudaMalloc / cudaFree: its per-CTA partial sums and its last-CTA ticket live
// in the file-scope array below, which every GPU that loads the library keeps
// until the process exits.
namespace gbf {
namespace {

constexpr int kStaticReduceCtas = 2048;  // 2048 CTAs x 1024 pixels: up to 2,097,152 pixels per image
constexpr int kStaticTicketSlot = kStaticReduceCtas * kPartialStride;

// partial records of kStaticReduceCtas CTAs, then the ticket (as unsigned bits)
static __device__ __align__(256) float g_reduce_scratch[kStaticTicketSlot + 64];

__global__ void __launch_bounds__(kReduceThreads, 3) reduce_static_kernel(SessionView sv, ReduceArgs a,
                                                                          float *scratch, double *out) {
    const int nctas = sv.red_ctas[0];
    __shared__ ReduceSmem sm;
    stage_ref_tile(sm, sv, 0, 0, blockIdx.x, kCtaPixels);
    __shared__ M34 T;
    __shared__ float huber_s;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < 12; ++i) T.m[i] = a.pose[i];
        huber_s = photo_huber(a.stddev);
    }
    __syncthreads();
    cta_partial<false>(sm, sv, 0, 0, 1, T, a.stddev, huber_s, blockIdx.x, kCtaPixels, scratch + (size_t)blockIdx.x * kPartialStride);
    __threadfence();
    __syncthreads();
    __shared__ unsigned int ticket;
    unsigned *tk = reinterpret_cast<unsigned *>(scratch + kStaticTicketSlot);
    if (threadIdx.x == 0) ticket = atomicAdd(tk, 1u);
    __syncthreads();
    if (ticket != (unsigned)nctas - 1u) return;
    __threadfence();
    __shared__ double total[kReduceWidth];
    sum_partials(sm, scratch, nctas, total);
    if (threadIdx.x < kReduceWidth) out[threadIdx.x] = total[threadIdx.x];
    if (threadIdx.x == 0) *tk = 0u;
}

// device address of g_reduce_scratch per device, looked up once with that device current
std::mutex g_scratch_mu;
float *g_scratch_ptr[64] = {};

gbf_status static_scratch(float **ptr) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_error(e, "gbf_reduce_noalloc: cudaGetDevice");
    if (dev < 0 || dev >= 64) return set_error(GBF_ERR_INVALID_ARG, "gbf_reduce_noalloc: device index >= 64");
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_reduce_scratch);
        if (e != cudaSuccess) return cuda_error(e, "gbf_reduce_noalloc: cudaGetSymbolAddress");
        g_scratch_ptr[dev] = static_cast<float *>(p);
    }
    *ptr = g_scratch_ptr[dev];
    return GBF_OK;
}

}  // namespace
}  // namespace gbf

extern "C" GBF_API gbf_status gbf_reduce_noalloc(const gbf_reduce_inputs *in, const double T[16], float stddev,
                                                 double *out_dev, void *stream) {
    using namespace gbf;
    if (!in || !T || !out_dev || !in->ref_vmap || !in->ref_nmap || !in->ref_intensity || !in->cur_vmap ||
        !in->cur_nmap || !in->cur_intensity || !in->cur_didx || !in->cur_didy)
        return set_error(GBF_ERR_INVALID_ARG, "gbf_reduce_noalloc: null pointer");
    if (in->width < 8 || in->height < 8 || !(in->fx > 0) || !(in->fy > 0))
        return set_error(GBF_ERR_INVALID_ARG, "gbf_reduce_noalloc: bad image size or focal length");
    // the reference images are staged in 16-byte copies, the vertex and normal
    // maps read as float4, the other images as float
    auto aligned = [](const void *p, uintptr_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
    if (!aligned(in->ref_vmap, 16) || !aligned(in->ref_nmap, 16) || !aligned(in->ref_intensity, 16) ||
        !aligned(in->cur_vmap, 16) || !aligned(in->cur_nmap, 16) || !aligned(in->cur_intensity, 4) ||
        !aligned(in->cur_didx, 4) || !aligned(in->cur_didy, 4))
        return set_error(GBF_ERR_INVALID_ARG,
                         "gbf_reduce_noalloc: vertex, normal and reference intensity images must be 16-byte aligned");
    if (!aligned(out_dev, 8))  // written as doubles
        return set_error(GBF_ERR_INVALID_ARG, "gbf_reduce_noalloc: out_dev must be 8-byte aligned");
    const long long pixels = (long long)in->width * in->height;
    if (pixels > (long long)kStaticReduceCtas * kReduceThreads * kReducePixelsPerThread)
        return set_error(GBF_ERR_CAPACITY, "gbf_reduce_noalloc: at most 2,097,152 pixels per image");
    float *scratch = nullptr;
    gbf_status st = static_scratch(&scratch);
    if (st != GBF_OK) return st;
    // a SessionView over the caller's level-0 images: set 0 = reference, set 1 = current
    SessionView sv;
    memset(&sv, 0, sizeof(sv));
    sv.levels = 1;
    LevelK &K = sv.lv[0];
    K.w = in->width; K.h = in->height;
    K.fx = in->fx; K.fy = in->fy; K.cx = in->cx; K.cy = in->cy;
    K.invfx = 1.0f / in->fx; K.invfy = 1.0f / in->fy;
    sv.red_ctas[0] = reduce_ctas((int)pixels);
    square_gates(sv, in->dist_thresh, in->angle_thresh);
    sv.vmap[0][0] = (float4 *)in->ref_vmap;
    sv.nmap[0][0] = (float4 *)in->ref_nmap;
    sv.inten[0][0] = (float *)in->ref_intensity;
    sv.vmap[1][0] = (float4 *)in->cur_vmap;
    sv.nmap[1][0] = (float4 *)in->cur_nmap;
    sv.inten[1][0] = (float *)in->cur_intensity;
    sv.gx[0] = (float *)in->cur_didx;
    sv.gy[0] = (float *)in->cur_didy;
    ReduceArgs a{};
    a.once = 1;
    for (int i = 0; i < 12; ++i) a.pose[i] = (float)T[i];
    a.stddev = stddev;
    cudaStream_t s = (cudaStream_t)stream;
    // the ticket must start at zero whatever an earlier, interrupted call left
    cudaError_t e = cudaMemsetAsync(scratch + kStaticTicketSlot, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return cuda_error(e, "gbf_reduce_noalloc: clear ticket");
    reduce_static_kernel<<<sv.red_ctas[0], kReduceThreads, 0, s>>>(sv, a, scratch, out_dev);
    return check_cuda("gbf_reduce_noalloc");
}
