// ingest.cu -- frame ingest and tracking pyramids (DeviceImage::upload,
// src/tracking/device_image.cpp:146-181; kernels of src/tracking/cuda_imgproc.cu).
//
// Two launches per frame for all sessions of a batch:
//   1. ingest:     u16 mm -> metres (System::process_images, src/system.cpp:43),
//                  rgb8 -> uchar4 + grey (device_image.cpp:161-162), bilateral
//                  filter of the tracking depth (cuda_imgproc.cu:197-200), and
//                  levels 1 and 2: 2x2 mean of depth (cv::cuda::resize 0.5,
//                  cuda_imgproc.cu:202-205) and 5x5 binomial pyrDown of the
//                  intensity (cuda_imgproc.cu:207-210), from shared-memory tiles.
//                  Levels 3 and 4, where configured, are a launch each (pyr_down).
//   2. level_maps: every level in one launch: dI/dx, dI/dy (computeDerivativeK,
//                  cuda_imgproc.cu:217-234), vertex map (backProjectDepthK,
//                  :249-263) and normal map (computeNMapK, :276-294), the normal
//                  computed from back-projected neighbours so no second pass.
// The OpenCV filters are third-party code absent here; they are restated from
// their documented definitions (bilateral: circular 5-tap window, Gaussian
// space/range weights; resize: pixel-centre bilinear at exactly 0.5; pyrDown:
// [1 4 6 4 1]/16 separable, reflect-101 border).
#include "gbf_device.cuh"
#include "gbf_kernels.h"

namespace gbf {

namespace {

__device__ __forceinline__ int reflect101(int i, int n) {
    if (i < 0) i = -i;
    if (i >= n) i = 2 * n - 2 - i;
    return i;
}

__device__ __forceinline__ int clamp_index(int i, int n) { return min(max(i, 0), n - 1); }

__device__ __forceinline__ int set_index(const SessionView &sv, int sel) {
    const int idx = sv.ts->idx;
    return sel ? idx : 1 - idx;
}

// The frame's images and its pyramid down to level 2, a CTA per 32x32 tile of level 0.
// Level 1 needs the grey image two pixels around the tile and level 2 level 1 two around
// its part, six pixels of level 0 together, which every CTA converts for itself
// (1.9 times the tile); the depth means stay within the tile.
// What bounds it: issue, most of it the bilateral filter's thirteen exponentials.
// A thread filters four rows of a column, whose windows share 28 of 52 samples, and the
// binomial runs along rows and then columns, a lane per column whose reflected indices it
// keeps.  As launches of their own (a pixel per thread, a window each; then a launch per
// level) the three levels took, and take here: 8 sessions of 640x480 53 -> 45 us, one of
// 1280x720 27 -> 21, of 320x240 12.4 -> 7.6.  40 or 48 registers instead of 64: 2% and 1% slower.
constexpr int kTile = 32, kTileRows = 4, kTileThreads = kTile * kTile / kTileRows, kTileWarps = kTileThreads / 32;
constexpr int kWin = 2, kGrey = 6;                                        // halos of the depth and the grey image
constexpr int kZ = kTile + 2 * kWin, kG = kTile + 2 * kGrey, kG1 = kTile / 2 + 4;
struct TileSmem {
    float z[kZ][kZ];               // depth
    float g[kG][kG];               // grey; read only where the image is
    float h[kG][kG1];              // its rows, filtered for level 1
    float g1[kG1][kG1];            // level 1, two pixels around the tile's part
    float f[kTile][kTile];         // filtered depth
    float d1[kTile / 2][kTile / 2];
};

__device__ __forceinline__ float binomial5(float a, float b, float c, float d, float e) {
    return (((a + 4.f * b) + 6.f * c) + 4.f * d) + e;
}

__global__ void __launch_bounds__(kTileThreads, 4) ingest_kernel(const SessionView *__restrict__ svs, IngestArgs a) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active) return;
    const int W = sv.lv[0].w, H = sv.lv[0].h, levels = sv.levels;
    const int tiles_x = (W + kTile - 1) / kTile;
    const int x0 = (blockIdx.x % tiles_x) * kTile, y0 = (blockIdx.x / tiles_x) * kTile;
    if (y0 >= H) return;  // uniform per CTA
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, set = set_index(sv, a.set_sel);
    __shared__ TileSmem sm;

    // the tile's depth and colour, all loads before the first store: a warp per row,
    // columns 0..31 of it, then what the halo adds
    constexpr int kZRows = (kZ + kTileWarps - 1) / kTileWarps, kGRows = (kG + kTileWarps - 1) / kTileWarps;
    float za[kZRows], zb[kZRows];
    {
        // (past the image's far border a tile holds samples that no pixel reads)
        const int xa = clamp_index(reflect101(x0 + lane - kWin, W), W);
        const int xb = clamp_index(reflect101(x0 + 32 + lane - kWin, W), W);
        const char *rows = a.src == 0 ? reinterpret_cast<const char *>(sv.in_depth) : static_cast<const char *>(a.depth);
        const long long pitch = a.src == 0 ? (long long)W * 2 : a.depth_pitch;
        const auto load = [&](const auto &at) {
#pragma unroll
            for (int k = 0; k < kZRows; ++k) {
                const int r = warp + k * kTileWarps;
                const char *row = rows + clamp_index(reflect101(y0 + r - kWin, H), H) * pitch;
                za[k] = zb[k] = 0.f;
                if (r < kZ) {
                    za[k] = at(row, xa);
                    if (lane < 2 * kWin) zb[k] = at(row, xb);
                }
            }
        };
        if (a.src == 2) load([](const char *row, int x) { return reinterpret_cast<const float *>(row)[x]; });
        else load([](const char *row, int x) { return (float)reinterpret_cast<const uint16_t *>(row)[x] * 0.001f; });
    }
    {
        const uint8_t *rgb = a.src == 0 ? sv.in_rgb : a.rgb;
        const long long pitch = a.src == 0 ? (long long)W * 3 : a.rgb_pitch;
        const int hx = lane < kGrey ? x0 - kGrey + lane : x0 + kTile + lane - kGrey;  // halo columns, lanes 0..11
        uchar4 ca[kGRows], cb[kGRows];
#pragma unroll
        for (int k = 0; k < kGRows; ++k) {
            const int r = warp + k * kTileWarps, y = y0 + r - kGrey;
            const bool in = r < kG && y >= 0 && y < H && (levels > 1 || (r >= kGrey && r < kGrey + kTile));
            const auto load = [&](int x) {
                const uint8_t *px = rgb + y * pitch + (long long)x * 3;
                return make_uchar4(px[0], px[1], px[2], 0);
            };
            ca[k] = cb[k] = make_uchar4(0, 0, 0, 0);
            if (in && x0 + lane < W) ca[k] = load(x0 + lane);
            if (in && levels > 1 && lane < 2 * kGrey && hx >= 0 && hx < W) cb[k] = load(hx);
        }
#pragma unroll
        for (int k = 0; k < kZRows; ++k) {
            const int r = warp + k * kTileWarps;
            if (r < kZ) {
                sm.z[r][lane] = za[k];
                if (lane < 2 * kWin) sm.z[r][32 + lane] = zb[k];
            }
        }
        // cv::COLOR_RGB2GRAY on CV_32FC3: 0.299 R + 0.587 G + 0.114 B
        const auto grey = [](uchar4 c) { return (0.299f * (float)c.x + 0.587f * (float)c.y) + 0.114f * (float)c.z; };
#pragma unroll
        for (int k = 0; k < kGRows; ++k) {
            const int r = warp + k * kTileWarps, y = y0 + r - kGrey;
            if (r >= kG) continue;
            const float v = grey(ca[k]);
            sm.g[r][kGrey + lane] = v;
            if (lane < 2 * kGrey) sm.g[r][lane < kGrey ? lane : kTile + lane] = grey(cb[k]);
            if (r >= kGrey && r < kGrey + kTile && y < H && x0 + lane < W) {
                const size_t p = (size_t)y * W + x0 + lane;
                sv.rgb4[p] = ca[k];
                sv.inten[set][0][p] = v;
            }
        }
    }
    __syncthreads();

    // depth: rows 4 warp .. + 3 of column lane
    {
        const int r0 = kTileRows * warp;
        float m[kTileRows + 4], l1[kTileRows + 2], r1[kTileRows + 2], l2[kTileRows], r2[kTileRows];
#pragma unroll
        for (int k = 0; k < kTileRows + 4; ++k) m[k] = sm.z[r0 + k][lane + 2];
#pragma unroll
        for (int k = 0; k < kTileRows + 2; ++k) {
            l1[k] = sm.z[r0 + k + 1][lane + 1];
            r1[k] = sm.z[r0 + k + 1][lane + 3];
        }
#pragma unroll
        for (int k = 0; k < kTileRows; ++k) {
            l2[k] = sm.z[r0 + k + 2][lane];
            r2[k] = sm.z[r0 + k + 2][lane + 4];
        }
#pragma unroll
        for (int k = 0; k < kTileRows; ++k) {
            const float c = m[k + 2];
            float filt = c;
            if (sv.bilateral) {
                // circular window of radius 2 (cv::cuda::bilateralFilter(src, dst, 5, 1, 1))
                const float ks = -0.5f, kc = -0.5f;  // -1/(2 sigma^2), sigma_space = sigma_colour = 1
                float s1 = 0.f, s2 = 0.f;
                const auto tap = [&](float v, int sp) {
                    const float d = v - c;
                    const float w = expf((float)sp * ks + (d * d) * kc);
                    s1 += w * v;
                    s2 += w;
                };
                tap(m[k], 4);
                tap(l1[k], 2); tap(m[k + 1], 1); tap(r1[k], 2);
                tap(l2[k], 4); tap(l1[k + 1], 1); tap(c, 0); tap(r1[k + 1], 1); tap(r2[k], 4);
                tap(l1[k + 2], 2); tap(m[k + 3], 1); tap(r1[k + 2], 2);
                tap(m[k + 4], 4);
                filt = s1 / s2;
            }
            sm.f[r0 + k][lane] = filt;
            const int y = y0 + r0 + k, x = x0 + lane;
            if (y < H && x < W) {
                const size_t p = (size_t)y * W + x;
                sv.depth_raw[p] = c;
                sv.depth[0][p] = filt;
            }
        }
    }
    if (levels < 2) return;
    const int w1 = sv.lv[1].w, h1 = sv.lv[1].h, X1 = x0 / 2, Y1 = y0 / 2;
    // intensity: 5x5 binomial, reflect-101, sample at (2x, 2y); its rows first, a warp
    // per row and a lane per column of level 1
    const int x1 = X1 - 2 + lane;
    const bool in1 = lane < kG1 && x1 >= 0 && x1 < w1;
    {
        const int at = 2 * x1, o = kGrey - x0;
        const int c0 = abs(at - 2) + o, c1 = abs(at - 1) + o, c3 = reflect101(at + 1, W) + o, c4 = reflect101(at + 2, W) + o;
        if (in1) {
#pragma unroll 2
            for (int r = warp; r < kG; r += kTileWarps) {
                const float *row = sm.g[r];
                sm.h[r][lane] = binomial5(row[c0], row[c1], row[at + o], row[c3], row[c4]);
            }
        }
    }
    __syncthreads();
    for (int r = warp; r < kG1; r += kTileWarps) {
        const int y = Y1 - 2 + r, at = 2 * y, o = kGrey - y0;
        if (!in1 || y < 0 || y >= h1) continue;
        const float v = binomial5(sm.h[abs(at - 2) + o][lane], sm.h[abs(at - 1) + o][lane], sm.h[at + o][lane],
                                  sm.h[reflect101(at + 1, H) + o][lane], sm.h[reflect101(at + 2, H) + o][lane]) *
                        (1.f / 256.f);
        sm.g1[r][lane] = v;
        if (r >= 2 && r < 2 + kTile / 2 && lane >= 2 && lane < 2 + kTile / 2) sv.inten[set][1][(size_t)y * w1 + x1] = v;
    }
    // depth: 2x2 mean (resize by 0.5, pixel-centre bilinear)
    const auto mean = [](float a0, float a1, float a2, float a3) { return (((a0 + a1) + a2) + a3) * 0.25f; };
    {
        const int lx = tid & 15, ly = tid >> 4, x = X1 + lx, y = Y1 + ly;
        if (x < w1 && y < h1) {
            const float v = mean(sm.f[2 * ly][2 * lx], sm.f[2 * ly][2 * lx + 1], sm.f[2 * ly + 1][2 * lx],
                                 sm.f[2 * ly + 1][2 * lx + 1]);
            sm.d1[ly][lx] = v;
            sv.depth[1][(size_t)y * w1 + x] = v;
        }
    }
    if (levels < 3) return;
    __syncthreads();
    const int w2 = sv.lv[2].w, h2 = sv.lv[2].h, lx = tid & 7, ly = (tid >> 3) & 7, x = x0 / 4 + lx, y = y0 / 4 + ly;
    if (x >= w2 || y >= h2) return;
    if (tid < 64) {
        float hrow[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            const float *row = sm.g1[reflect101(2 * y + j - 2, h1) - (Y1 - 2)] + (2 - X1);
            const int at = 2 * x;
            hrow[j] = binomial5(row[abs(at - 2)], row[abs(at - 1)], row[at], row[reflect101(at + 1, w1)],
                                row[reflect101(at + 2, w1)]);
        }
        sv.inten[set][2][(size_t)y * w2 + x] = binomial5(hrow[0], hrow[1], hrow[2], hrow[3], hrow[4]) * (1.f / 256.f);
    } else if (tid < 128) {
        sv.depth[2][(size_t)y * w2 + x] =
            mean(sm.d1[2 * ly][2 * lx], sm.d1[2 * ly][2 * lx + 1], sm.d1[2 * ly + 1][2 * lx], sm.d1[2 * ly + 1][2 * lx + 1]);
    }
}

// Levels 3 and up, a launch each.
__global__ void pyr_down_kernel(const SessionView *__restrict__ svs, int set_sel, int level) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active || level >= sv.levels) return;
    const int w = sv.lv[level].w, h = sv.lv[level].h;
    const int pw = sv.lv[level - 1].w, ph = sv.lv[level - 1].h;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * h) return;
    const int x = i % w, y = i / w;
    const int set = set_index(sv, set_sel);

    // depth: 2x2 mean (resize by 0.5, pixel-centre bilinear)
    const float *sd = sv.depth[level - 1];
    const float a0 = sd[(size_t)(2 * y) * pw + 2 * x], a1 = sd[(size_t)(2 * y) * pw + 2 * x + 1];
    const float a2 = sd[(size_t)(2 * y + 1) * pw + 2 * x], a3 = sd[(size_t)(2 * y + 1) * pw + 2 * x + 1];
    sv.depth[level][i] = (((a0 + a1) + a2) + a3) * 0.25f;

    // intensity: 5x5 binomial, reflect-101, sample at (2x, 2y)
    const float *si = sv.inten[set][level - 1];
    int xs[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) xs[k] = reflect101(2 * x + k - 2, pw);
    float hrow[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const float *row = si + (size_t)reflect101(2 * y + j - 2, ph) * pw;
        hrow[j] = (((row[xs[0]] + 4.f * row[xs[1]]) + 6.f * row[xs[2]]) + 4.f * row[xs[3]]) + row[xs[4]];
    }
    sv.inten[set][level][i] = ((((hrow[0] + 4.f * hrow[1]) + 6.f * hrow[2]) + 4.f * hrow[3]) + hrow[4]) * (1.f / 256.f);
}

// backProjectDepthK (cuda_imgproc.cu:249-263)
__device__ __forceinline__ float4 back_project(float z, int x, int y, const LevelK &K) {
    if (z > 0.3f && z < 5.0f)
        return make_float4((z * ((float)x - K.cx)) * K.invfx, (z * ((float)y - K.cy)) * K.invfy, z, 1.0f);
    return make_float4(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff), __int_as_float(0x7fffffff), -1.0f);
}

__device__ __forceinline__ float4 normal_from(float4 v00, float4 v01, float4 v10, float4 v11) {
    const float3 a = make_float3(v01.x - v00.x, v01.y - v00.y, v01.z - v00.z);
    const float3 b = make_float3(v11.x - v10.x, v11.y - v10.y, v11.z - v10.z);
    const float3 n = cross3(a, b);
    const float l = norm3(n.x, n.y, n.z);
    return make_float4(n.x / l, n.y / l, n.z / l, 1.f);
}

// Integration test and weight of the frame's pixel for the normal-weighted
// update (update_map_weighted_kernel, depth_fusion.cu:390-405): raw depth `dist`,
// level-0 normal of the filtered depth; rejected pixels carry NaN depth.
__device__ __forceinline__ float2 fuse_weight(const SessionView &sv, float dist, float4 n) {
    const bool ok = !(isnan(dist) || isnan(n.x) || dist > sv.zmax_u || dist < sv.zmin_u);
    const float w = fabsf(sinf(n.z)) / (dist * dist);
    return make_float2(ok ? dist : __int_as_float(0x7fffffff), w);
}

// Every level's vertex, normal, gradient and packed images, a thread per strip of
// kMapRows pixels of a column.  A pixel needs itself and four neighbours of two
// images: a strip of four loads 28 values, all in flight at once, where a pixel per
// thread loaded 10 each and waited with 28% of them in L1; the stores of a warp stay rows.
// Its bytes then bound it (8 sessions of 640x480: 56 -> 42 us, 6.2 TB/s written and
// read; one of 1280x720 18.4 -> 15.5).  Strips of two 52 us, 64 registers 43.
constexpr int kMapRows = 4, kMapThreads = 256;
__host__ __device__ inline int map_ctas(int w, int h) {
    return (w * ((h + kMapRows - 1) / kMapRows) + kMapThreads - 1) / kMapThreads;
}
__global__ void __launch_bounds__(kMapThreads, 3) level_maps_kernel(const SessionView *__restrict__ svs, int set_sel) {
    chain_begin();
    const SessionView &sv = svs[blockIdx.y];
    if (!sv.active) return;
    // flatten the levels
    int b = blockIdx.x, level = 0;
    for (; level < sv.levels; ++level) {
        const int n = map_ctas(sv.lv[level].w, sv.lv[level].h);
        if (b < n) break;
        b -= n;
    }
    if (level >= sv.levels) return;
    const LevelK K = sv.lv[level];
    const int i = b * kMapThreads + threadIdx.x;
    const int strip = i / K.w, x = i - strip * K.w, y0 = strip * kMapRows;
    if (y0 >= K.h) return;
    const int set = set_index(sv, set_sel);
    const float *__restrict__ I = sv.inten[set][level];
    const float *__restrict__ D = sv.depth[level];
    const bool fuse = level == 0 && set_sel == 0;

    const int xl = max(x - 1, 0), xr = min(x + 1, K.w - 1);
    float dc[kMapRows + 2], ic[kMapRows + 2];  // the column, one row above to one below
    float dl[kMapRows], dr[kMapRows], il[kMapRows], ir[kMapRows], raw[kMapRows];
#pragma unroll
    for (int k = 0; k < kMapRows + 2; ++k) {
        const int at = min(max(y0 + k - 1, 0), K.h - 1) * K.w + x;
        dc[k] = D[at];
        ic[k] = I[at];
    }
#pragma unroll
    for (int k = 0; k < kMapRows; ++k) {
        const int row = min(y0 + k, K.h - 1) * K.w;
        dl[k] = D[row + xl];
        dr[k] = D[row + xr];
        il[k] = I[row + xl];
        ir[k] = I[row + xr];
        raw[k] = fuse ? sv.depth_raw[row + x] : 0.f;
    }
    float *gxs = sv.gx[level], *gys = sv.gy[level];
    float4 *igd = sv.igd[set][level], *nmap = sv.nmap[set][level], *vmap = sv.vmap[set][level];
    const float nanf_ = __int_as_float(0x7fffffff);
    float4 up = back_project(dc[0], x, max(y0 - 1, 0), K), here = back_project(dc[1], x, y0, K);
#pragma unroll
    for (int k = 0; k < kMapRows; ++k) {
        const int y = y0 + k;
        if (y >= K.h) break;
        const float4 down = back_project(dc[k + 2], x, y + 1, K);
        // the reference leaves the last row / column unwritten; write invalid
        float gx = 0.f, gy = 0.f;
        float4 n = make_float4(nanf_, nanf_, nanf_, nanf_);
        if (x < K.w - 1 && y < K.h - 1) {
            gx = (ir[k] - il[k]) * 0.5f;
            gy = (ic[k + 2] - ic[k]) * 0.5f;
            n = normal_from(back_project(dl[k], xl, y, K), back_project(dr[k], x + 1, y, K), up, down);
        }
        const int at = y * K.w + x;
        gxs[at] = gx;
        gys[at] = gy;
        igd[at] = make_float4(ic[k + 1], gx, gy, 0.f);
        nmap[at] = n;
        vmap[at] = here;
        if (fuse) sv.fuse_px[at] = fuse_weight(sv, raw[k], n);
        up = here;
        here = down;
    }
}

}  // namespace

void launch_ingest(const SessionView *d_sv, int nslots, const Extent &ex, const IngestArgs &a, cudaStream_t st) {
    const int tiles = ((ex.w + kTile - 1) / kTile) * ((ex.h + kTile - 1) / kTile);
    launch_kernel(ingest_kernel, dim3(tiles, nslots), kTileThreads, ex.chain, st, d_sv, a);
    int w = ex.w / 4, h = ex.h / 4;
    for (int l = 3; l < ex.levels; ++l) {
        w /= 2; h /= 2;
        launch_kernel(pyr_down_kernel, dim3((w * h + 255) / 256, nslots), 256, ex.chain, st, d_sv, a.set_sel, l);
    }
    int total = 0;
    w = ex.w; h = ex.h;
    for (int l = 0; l < ex.levels; ++l) {
        total += map_ctas(w, h);
        w /= 2; h /= 2;
    }
    launch_kernel(level_maps_kernel, dim3(total, nslots), kMapThreads, ex.chain, st, d_sv, a.set_sel);
}

}  // namespace gbf
