// gn_step.cuh -- the Gauss-Newton step in FP64, spread over one warp: the 6x6
// LDL^T with symmetric diagonal pivoting (the documented method of Eigen::LDLT
// used at icp_tracker.cpp:92; zero pivots act as a pseudo-inverse), the SE(3)
// exponential of xi = (rho, phi), translation first (Sophus convention), and
// the pose composition.
//
// What bounds it: a GB300 SM issues one FP64 instruction of a warp every 64
// cycles, dependent or not and whatever number of its lanes is active (measured
// with clock64: 64 fused multiply-adds, one chain or eight, take 64 x 64 cycles
// with 1 or 32 lanes; a division takes 580, a square root 590, sincos 1,620,
// rcp.approx.ftz.f64 24).  So the step's time is its count of FP64 instructions,
// and lanes are free: the right-hand side is a seventh row of the matrix and is
// eliminated with it, a pivot costs one reciprocal (three fused multiply-adds)
// that every lane multiplies by instead of a division, the pivot search runs on
// the bit patterns in the integer pipe, the back substitution takes one
// instruction per unknown for all the rows that remain, and the exponential's
// coefficients are series evaluated for all three in the same instructions.
// Selects stand in place of lane-dependent branches throughout: where the
// compiler does not join a warp again after one, every FP64 instruction that
// follows is issued once per part (seen as 4 to 8 times the cycles).
// Measured in the reduction's last CTA, one 640x480 session (clock64): the solve
// 21,000 -> 4,500 cycles, the exponential and the composition 8,300 -> 2,400.  Of
// these 6,900 the 35 and 17 FP64 instructions hold 3,330; the rest is shuffles, the
// pivot search, index arithmetic and the loops.
#pragma once

#include <cuda_runtime.h>

#include "gbf_types.h"

namespace gbf {

// Full-warp shuffles: every lane must reach each call (none may sit inside a
// lane-dependent branch or operand).
__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
// lane holding the unordered pair {a, b} of a symmetric 6x6 matrix (lower
// triangle, lanes 0..20; row 6, lanes 21..26, is the right-hand side)
__device__ __forceinline__ int tri6(int a, int b) { return a >= b ? a * (a + 1) / 2 + b : b * (b + 1) / 2 + a; }
// its row, without a loop: lanes that left a loop at different trips would run
// what follows one group after the other where the compiler does not join them
__device__ __forceinline__ int tri_row(int lane) {
    return (lane >= 1) + (lane >= 3) + (lane >= 6) + (lane >= 10) + (lane >= 15) + (lane >= 21);
}
constexpr unsigned kDiagLanes = 0x104225u;  // lanes 0, 2, 5, 9, 14, 20

// 1 / d to about one unit in the last place, 0 for an infinity: the hardware's
// approximation (20 bits) and one third-order Householder step, whose error is
// the cube of its input's.  For 2^-959 <= |d| <= 2^959: the matrices are made of floats, and no
// elimination of them leaves a pivot outside that (a difference is a multiple of
// an operand's last place).
__device__ __forceinline__ double recip_d(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = __fma_rn(-d, y, 1.0);
    const double v = __fma_rn(y, __fma_rn(e, e, e), y);
    return (__double2hiint(d) & 0x7fffffff) == 0x7ff00000 && __double2loint(d) == 0 ? 0.0 : v;
}

// x = A^-1 b.  In: lane tri6(r, c) holds A[r][c] (r >= c, r < 6) and lane 21 + c
// holds b[c], c < 6.  Out: lane 21 + c holds x[c].  The pivoting moves nothing:
// the lanes keep original indices and a mask of the pivots taken.  (Without the
// search the same elimination takes 3,600 cycles instead of 3,760: the reciprocals hide it.)
__device__ __forceinline__ double ldlt_solve6_warp(double a) {
    const int lane = threadIdx.x & 31;
    const int r = lane < 27 ? tri_row(lane) : 0, c = lane < 27 ? lane - r * (r + 1) / 2 : 0;
    __syncwarp();
    unsigned done = 0;   // bit i: index i has been the pivot
    unsigned order = 0;  // the pivots in turn, four bits each
#pragma unroll 1
    for (int k = 0; k < 6; ++k) {
        // each element's reciprocal beside the search for the pivot, whose lane has
        // it then: the remaining diagonal element of the largest magnitude by the
        // high word of its bit pattern (a tie there, to 2^-20, goes to the lowest index)
        const double own = recip_d(a);
        const unsigned mag = (unsigned)__double2hiint(a) & 0x7fffffffu;
        const bool cand = ((kDiagLanes >> lane) & 1u) && !((done >> r) & 1u);
        const unsigned top = __reduce_max_sync(0xffffffffu, cand ? mag : 0u);
        const int src = __ffs(__ballot_sync(0xffffffffu, cand && mag == top)) - 1;
        const int p = __popc(kDiagLanes & ((1u << src) - 1u));
        const double D = shfl_d(a, src), inv = shfl_d(own, src);
        const double ar = shfl_d(a, tri6(r, p)), ac = shfl_d(a, tri6(c, p));
        done |= 1u << p;
        order |= (unsigned)p << (4 * k);
        // rows and columns still to be eliminated (row 6 always is), and the pivot's own column
        const bool rest_r = !((done >> r) & 1u), rest_c = !((done >> c) & 1u);
        const bool inner = rest_r && rest_c, column = (c == p && rest_r) || (r == p && rest_c);
        // selects, not branches: every lane stays with the warp.  |D| <= DBL_MIN: no
        // contribution of this unknown (L = 0)
        const unsigned dh = (unsigned)__double2hiint(D) & 0x7fffffffu;
        const bool zero = dh < 0x00100000u || (dh == 0x00100000u && __double2loint(D) == 0);
        const double t = (r == p ? a : ar) * inv;
        const double L = zero ? 0.0 : t;
        const double next = __fma_rn(-L, ac, a);
        a = inner ? next : column ? L : a;
    }
    // back substitution, last pivot first: the rows whose pivots came earlier take their term at once
#pragma unroll 1
    for (int k = 5; k > 0; --k) {
        const int q = (order >> (4 * k)) & 15u;
        done &= ~(1u << q);
        const double x = shfl_d(a, 21 + q), L = shfl_d(a, tri6(c, q));
        const double next = __fma_rn(-L, x, a);
        a = r == 6 && ((done >> c) & 1u) ? next : a;
    }
    return a;
}

// element idx of W = [w]x (row-major 3x3)
__device__ __forceinline__ double skew_at(int idx, double wx, double wy, double wz) {
    return idx == 1 ? -wz : idx == 2 ? wy : idx == 3 ? wz : idx == 5 ? -wx : idx == 6 ? -wy : idx == 7 ? wx : 0.0;
}

// the coefficients in closed form, out of line: steps above 1/4 rad are rare, and
// inlined the trigonometry's branches and stack sit in every caller
__device__ __noinline__ static double exp_coefficient(double th2, int lane) {
    const double th = sqrt(th2);
    double s, co;
    sincos(th, &s, &co);
    return (lane == 0 ? s : lane == 1 ? 1.0 - co : th - s) / (lane == 0 ? th : lane == 1 ? th2 : th2 * th);
}

// exp(xi) T: lane 21 + c holds xi[c]; lane p = 4 i + j < 12 holds column j of T
// in (t0, t1, t2) and gets element (i, j) of the product.
__device__ __forceinline__ double se3_exp_mul_warp(double xi, double t0, double t1, double t2) {
    const int lane = threadIdx.x & 31;
    const double x0 = shfl_d(xi, 21), x1 = shfl_d(xi, 22), x2 = shfl_d(xi, 23);
    const double wx = shfl_d(xi, 24), wy = shfl_d(xi, 25), wz = shfl_d(xi, 26);
    const double th2 = __fma_rn(wz, wz, __fma_rn(wy, wy, wx * wx));
    // A = sin t / t, B = (1 - cos t) / t^2, C = (t - sin t) / t^3 on lanes 0, 1, 2
    double q;
    if (th2 < 0.0625) {
        // sum (-t^2)^n / (2 n + 1)!, (2 n + 2)!, (2 n + 3)!: the seven terms leave less than 1e-18
        // below 1/4 rad, beyond any step of a tracked frame
        const double x = -th2;
        auto pick = [&](double a, double b, double c) { return lane == 0 ? a : lane == 1 ? b : c; };
        q = pick(1.0 / 6227020800.0, 1.0 / 87178291200.0, 1.0 / 1307674368000.0);
        q = __fma_rn(q, x, pick(1.0 / 39916800.0, 1.0 / 479001600.0, 1.0 / 6227020800.0));
        q = __fma_rn(q, x, pick(1.0 / 362880.0, 1.0 / 3628800.0, 1.0 / 39916800.0));
        q = __fma_rn(q, x, pick(1.0 / 5040.0, 1.0 / 40320.0, 1.0 / 362880.0));
        q = __fma_rn(q, x, pick(1.0 / 120.0, 1.0 / 720.0, 1.0 / 5040.0));
        q = __fma_rn(q, x, pick(1.0 / 6.0, 1.0 / 24.0, 1.0 / 120.0));
        q = __fma_rn(q, x, pick(1.0, 0.5, 1.0 / 6.0));
    } else {
        q = exp_coefficient(th2, lane);
    }
    __syncwarp();
    // lanes 0..8: element e = (i, j) of R = I + A W + B W^2; lanes 9..17: of V = I + B W + C W^2;
    // W^2 = w w^T - t^2 I
    const bool rot = lane < 9;
    const int e = rot ? lane : lane < 18 ? lane - 9 : 0, i = e / 3, j = e % 3;
    const double f = shfl_d(q, rot ? 0 : 1), g = shfl_d(q, rot ? 1 : 2);
    const double wi = i == 0 ? wx : i == 1 ? wy : wz, wj = j == 0 ? wx : j == 1 ? wy : wz;
    const double w2 = __fma_rn(wi, wj, i == j ? -th2 : 0.0);
    const double m = __fma_rn(g, w2, __fma_rn(f, skew_at(e, wx, wy, wz), i == j ? 1.0 : 0.0));
    // lanes 0..11: row i of R times column j of T; lanes 12..14: row of V times rho, in the same instructions
    const bool tr = lane >= 12;
    const int row = tr ? (lane < 15 ? 9 + 3 * (lane - 12) : 9) : 3 * (lane / 4);
    const double m0 = shfl_d(m, row), m1 = shfl_d(m, row + 1), m2 = shfl_d(m, row + 2);
    const double v = __fma_rn(m2, tr ? x2 : t2, __fma_rn(m1, tr ? x1 : t1, m0 * (tr ? x0 : t0)));
    const double rho = shfl_d(v, 12 + (lane < 12 ? lane / 4 : 0));
    return (lane & 3) == 3 ? v + rho : v;
}

// 3x4 rigid transforms over a warp, lane p = 4 i + j < 12 holding element (i, j);
// the operations and their order are those of pose_inverse and pose_mul.
__device__ __forceinline__ double pose_inverse_warp(double e) {
    const int lane = threadIdx.x & 31, i = lane < 12 ? lane / 4 : 0, j = lane & 3;
    const double a0 = shfl_d(e, i), a1 = shfl_d(e, 4 + i), a2 = shfl_d(e, 8 + i);
    const double t0 = shfl_d(e, 3), t1 = shfl_d(e, 7), t2 = shfl_d(e, 11);
    const double t = -((a0 * t0 + a1 * t1) + a2 * t2);
    return j == 0 ? a0 : j == 1 ? a1 : j == 2 ? a2 : t;
}
__device__ __forceinline__ double pose_mul_warp(double a, double b) {
    const int lane = threadIdx.x & 31, i = lane < 12 ? lane / 4 : 0, j = lane & 3;
    const double a0 = shfl_d(a, 4 * i), a1 = shfl_d(a, 4 * i + 1), a2 = shfl_d(a, 4 * i + 2), a3 = shfl_d(a, 4 * i + 3);
    const double b0 = shfl_d(b, j), b1 = shfl_d(b, 4 + j), b2 = shfl_d(b, 8 + j);
    const double s = (a0 * b0 + a1 * b1) + a2 * b2;
    return j == 3 ? s + a3 : s;
}

// A pose as a kernel argument: no copy and no launch of its own.
struct MapPose {
    double p[12];
};

// The mapping pose and its float forms (update_map_floats), by one warp.
__device__ __forceinline__ void store_map_pose(TrackState *ts, const MapPose &pose) {
    const int lane = threadIdx.x & 31;
    double v = 0.0;
#pragma unroll
    for (int i = 0; i < 12; ++i)
        if (lane == i) v = pose.p[i];
    __syncwarp();
    const double inv = pose_inverse_warp(v);
    if (lane < 12) {
        ts->map_pose[lane] = v;
        ts->map_twc[lane] = (float)v;
        ts->map_tcw[lane] = (float)inv;
    }
}

}  // namespace gbf
