// Drives sessions through the C API and reaches into one's arena for what no
// caller can set: the numbers of the tracking run's words and the longest wait of
// its CTA 0 (csrc/tracking.cu).
// Prints what differs and returns 1, or returns 0.
#include <cuda.h>

#include <chrono>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../libfusion_gb300/csrc/gbf_internal.h"

using namespace gbf;

#define OK(call)                                                    \
    do {                                                            \
        if ((call) != 0) {                                          \
            printf("%s: %s\n", #call, gbf_last_error());            \
            return 1;                                               \
        }                                                           \
    } while (0)

constexpr int kW = 320, kH = 240;

struct Frames {
    gbf_synth_scene *sc = nullptr;
    gbf_intrinsics K{};
    uint16_t *depth = nullptr;
    uint8_t *rgb = nullptr;
    int open() {
        gbf_synth_params p;
        OK(gbf_synth_default(&p));
        OK(gbf_synth_create(&p, &sc));
        K.width = kW;
        K.height = kH;
        K.fx = K.fy = 262.5f;
        K.cx = 159.5f;
        K.cy = 119.5f;
        OK(cudaMalloc(&depth, kW * kH * 2));
        OK(cudaMalloc(&rgb, kW * kH * 3));
        return 0;
    }
    int render(int k) {
        double T[16];
        OK(gbf_synth_pose(sc, k, T));
        OK(gbf_synth_render(sc, &K, T, k, depth, rgb, nullptr));
        return 0;
    }
    int session(gbf_session **s) {
        gbf_config c;
        OK(gbf_config_default(&c));
        c.zmax_update = c.zmax_raycast = 4.f;
        c.num_buckets = 1 << 16;
        c.num_blocks = 1 << 14;
        OK(gbf_session_create(&c, &K, s));
        double T[16];
        OK(gbf_synth_pose(sc, 0, T));
        OK(gbf_set_pose(*s, T, nullptr));
        return 0;
    }
};

// Frames of a session whose run numbers start at `number` give those of a new one.
int numbers(Frames &f, unsigned number) {
    gbf_session *a, *b;
    if (f.session(&a) || f.session(&b)) return 1;
    const std::vector<unsigned long long> words((b->lay.total - b->lay.track_rec) / 8, (unsigned long long)number << 32);
    OK(cudaMemcpy(b->view.track_rec, words.data(), words.size() * 8, cudaMemcpyHostToDevice));
    OK(cudaMemcpy(b->view.ctr + C_TRACK_PUB, words.data(), 14 * 8, cudaMemcpyHostToDevice));
    for (int k = 0; k < 6; ++k) {
        if (f.render(k)) return 1;
        gbf_frame_stats x, y;
        double p[16], q[16];
        for (gbf_session *s : {a, b}) OK(gbf_process_frame(s, f.depth, kW * 2, f.rgb, kW * 3, nullptr));
        OK(gbf_get_pose(a, p, nullptr));
        OK(gbf_get_pose(b, q, nullptr));
        OK(gbf_get_stats(a, &x, nullptr));
        OK(gbf_get_stats(b, &y, nullptr));
        if (memcmp(p, q, sizeof(p)) || x.status || y.status || x.pixel_iterations != y.pixel_iterations) {
            printf("numbers from %#x, frame %d: status %u %u\n", number, k, x.status, y.status);
            return 1;
        }
    }
    OK(gbf_session_destroy(a));
    OK(gbf_session_destroy(b));
    return 0;
}

int set_wait(gbf_session *s, long long ns) {
    OK(cudaMemcpy(reinterpret_cast<char *>(s->d_view) + offsetof(SessionView, track_wait_ns), &ns, sizeof(ns),
                  cudaMemcpyHostToDevice));
    return 0;
}

// Runs whose CTA 0 does not wait at all (it gives up on the CTAs' arrival or on the
// first records): each ends at once, is told apart and leaves the next run as it was.
int lost(Frames &f) {
    gbf_session *s;
    if (f.session(&s)) return 1;
    for (int k = 0; k < 3; ++k) {
        if (f.render(k)) return 1;
        OK(gbf_process_frame(s, f.depth, kW * 2, f.rgb, kW * 3, nullptr));
    }
    double I[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1}, before[16], after[16];
    gbf_track_result want{}, got{};
    gbf_frame_stats st;
    OK(gbf_track(s, I, &want, nullptr));
    OK(gbf_get_stats(s, &st, nullptr));
    if (!want.success || want.iterations < 5 || st.status) {
        printf("success %d, %d iterations, status %u\n", want.success, want.iterations, st.status);
        return 1;
    }
    const auto t0 = std::chrono::steady_clock::now();
    for (int k = 0; k < 300; ++k) {
        if (set_wait(s, 0)) return 1;
        OK(gbf_track(s, I, &got, nullptr));
        OK(gbf_get_stats(s, &st, nullptr));
        if (got.success || memcmp(got.update, I, sizeof(I)) || st.status != GBF_FLAG_TRACK_WAIT) {
            printf("lost run %d: success %d, status %u\n", k, got.success, st.status);
            return 1;
        }
        if (set_wait(s, kTrackWaitNs)) return 1;
        OK(gbf_track(s, I, &got, nullptr));
        if (memcmp(&got, &want, sizeof(got))) {
            printf("the run after lost run %d: success %d, %d iterations\n", k, got.success, got.iterations);
            return 1;
        }
    }
    const double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (secs > 2.0) {  // one wait that ran its two seconds out
        printf("600 runs took %.3f s\n", secs);
        return 1;
    }
    // a frame: the pose stays, and the frame counts as not tracked
    OK(gbf_get_pose(s, before, nullptr));
    if (f.render(3) || set_wait(s, 0)) return 1;
    OK(gbf_process_frame(s, f.depth, kW * 2, f.rgb, kW * 3, nullptr));
    OK(gbf_get_pose(s, after, nullptr));
    OK(gbf_get_stats(s, &st, nullptr));
    if (memcmp(before, after, sizeof(before)) || st.track.success || st.status != (GBF_FLAG_TRACK_WAIT | GBF_FLAG_TRACK_FAILED)) {
        printf("frame: success %d, status %u\n", st.track.success, st.status);
        return 1;
    }
    OK(gbf_session_destroy(s));
    return 0;
}

// A stream of a green context with a few of the SMs, on which the run's CTAs do not fit
// at once: the frames are those of a stream with all of them.
int few_sms(Frames &f) {
    CUdevResource all{}, few{}, rest{};
    CUdevResourceDesc desc{};
    CUgreenCtx ctx{};
    CUstream st{};
    unsigned groups = 1;
    OK(cuDeviceGetDevResource(0, &all, CU_DEV_RESOURCE_TYPE_SM));
    OK(cuDevSmResourceSplitByCount(&few, &groups, &all, &rest, 0, 16));
    OK(cuDevResourceGenerateDesc(&desc, &few, 1));
    OK(cuGreenCtxCreate(&ctx, desc, 0, CU_GREEN_CTX_DEFAULT_STREAM));
    OK(cuGreenCtxStreamCreate(&st, ctx, CU_STREAM_NON_BLOCKING, 0));
    if (few.sm.smCount >= all.sm.smCount) {
        printf("%u of %u SMs\n", few.sm.smCount, all.sm.smCount);
        return 1;
    }
    gbf_session *a, *b;
    if (f.session(&a) || f.session(&b)) return 1;
    for (int k = 0; k < 4; ++k) {
        if (f.render(k)) return 1;
        OK(cudaDeviceSynchronize());
        gbf_frame_stats x, y;
        double p[16], q[16];
        OK(gbf_process_frame(a, f.depth, kW * 2, f.rgb, kW * 3, nullptr));
        OK(gbf_process_frame(b, f.depth, kW * 2, f.rgb, kW * 3, st));
        OK(gbf_get_pose(a, p, nullptr));
        OK(gbf_get_pose(b, q, st));
        OK(gbf_get_stats(a, &x, nullptr));
        OK(gbf_get_stats(b, &y, st));
        if (memcmp(p, q, sizeof(p)) || x.status || y.status || x.pixel_iterations != y.pixel_iterations) {
            printf("%u of %u SMs, frame %d: status %u %u\n", few.sm.smCount, all.sm.smCount, k, x.status, y.status);
            return 1;
        }
    }
    OK(gbf_session_destroy(a));
    OK(gbf_session_destroy(b));
    OK(cuStreamDestroy(st));
    OK(cuGreenCtxDestroy(ctx));
    return 0;
}

int main(int argc, char **argv) {
    Frames f;
    if (argc < 2 || f.open()) return 1;
    if (!strcmp(argv[1], "numbers")) return numbers(f, 5u) || numbers(f, 0x7ffffff5u) || numbers(f, 0xfffffff5u);
    if (!strcmp(argv[1], "lost")) return lost(f);
    if (!strcmp(argv[1], "few_sms")) return few_sms(f);
    return 1;
}
