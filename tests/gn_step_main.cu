// Runs the Gauss-Newton step's warp routines on cases from stdin: 27 doubles
// (lower triangle, right-hand side), 12 doubles (3x4 pose) each; writes the
// solution (6 doubles) and exp(x) T (12 doubles) of each.
#include <cstdio>
#include <vector>

#include "../libfusion_gb300/csrc/gn_step.cuh"

__global__ void run(const double *in, double *out) {
    const int lane = threadIdx.x;
    const double *p = in + blockIdx.x * 39;
    const double x = gbf::ldlt_solve6_warp(lane < 27 ? p[lane] : 0.0);
    const double *T = p + 27;
    const int j = lane & 3;
    const double e = gbf::se3_exp_mul_warp(x, T[j], T[4 + j], T[8 + j]);
    if (lane >= 21 && lane < 27) out[blockIdx.x * 18 + lane - 21] = x;
    if (lane < 12) out[blockIdx.x * 18 + 6 + lane] = e;
}

int main() {
    std::vector<double> h(39 * 4096), o;
    const size_t n = fread(h.data(), 39 * 8, 4096, stdin);
    double *in, *out;
    if (!n || cudaMalloc(&in, n * 39 * 8) != cudaSuccess || cudaMalloc(&out, n * 18 * 8) != cudaSuccess) return 1;
    cudaMemcpy(in, h.data(), n * 39 * 8, cudaMemcpyHostToDevice);
    run<<<(unsigned)n, 32>>>(in, out);
    o.resize(n * 18);
    if (cudaMemcpy(o.data(), out, n * 18 * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    return fwrite(o.data(), 18 * 8, n, stdout) == n ? 0 : 1;
}
