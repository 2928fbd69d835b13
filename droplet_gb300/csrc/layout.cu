// layout.cu -- conversion between the device layout of the populations
// (structure of arrays, f[i][z][y][x]) and the reference's host layout
// f_procs(1:15,x,y,z) (direction index fastest), used for checkpoints
// (outputfg, program/lbm_drop_xy.f90:721-743) and for resume / precursor reads
// (program/lbm_drop_xy.f90:789-823).
#include "dl_internal.cuh"

namespace dl {

// a block's sites through shared memory: both sides are read and written as runs
// (the strided side alone touched eight times its sectors)
constexpr int LAYOUT_NT = 128;

__global__ void __launch_bounds__(LAYOUT_NT) soa_to_aos_kernel(const double* __restrict__ soa, double* __restrict__ aos,
                                                               long long N) {
    __shared__ double buf[LAYOUT_NT * Q];
    const long long s0 = blockIdx.x * (long long)LAYOUT_NT, s = s0 + threadIdx.x;
    if (s < N) {
#pragma unroll
        for (int i = 0; i < Q; ++i) buf[threadIdx.x * Q + i] = __ldg(soa + i * N + s);
    }
    __syncthreads();
    const int n = (int)min((long long)LAYOUT_NT, N - s0) * Q;
    for (int t = threadIdx.x; t < n; t += LAYOUT_NT) aos[s0 * Q + t] = buf[t];
}

__global__ void __launch_bounds__(LAYOUT_NT) aos_to_soa_kernel(const double* __restrict__ aos, double* __restrict__ soa,
                                                               long long N) {
    __shared__ double buf[LAYOUT_NT * Q];
    const long long s0 = blockIdx.x * (long long)LAYOUT_NT, s = s0 + threadIdx.x;
    const int n = (int)min((long long)LAYOUT_NT, N - s0) * Q;
    for (int t = threadIdx.x; t < n; t += LAYOUT_NT) buf[t] = __ldg(aos + s0 * Q + t);
    __syncthreads();
    if (s >= N) return;
#pragma unroll
    for (int i = 0; i < Q; ++i) soa[i * N + s] = buf[threadIdx.x * Q + i];
}

static unsigned layout_blocks(const dl_handle* h) { return (unsigned)((h->N + LAYOUT_NT - 1) / LAYOUT_NT); }

int soa_to_aos(dl_handle* h, const double* d_soa, double* d_aos) {
    DL_LAUNCH(h, false, soa_to_aos_kernel<<<layout_blocks(h), LAYOUT_NT, 0, h->stream>>>(d_soa, d_aos, (long long)h->N));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

int aos_to_soa(dl_handle* h, const double* d_aos, double* d_soa) {
    DL_LAUNCH(h, false, aos_to_soa_kernel<<<layout_blocks(h), LAYOUT_NT, 0, h->stream>>>(d_aos, d_soa, (long long)h->N));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

__global__ void fill_kernel(double* __restrict__ d, double v, long long n) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t < n) d[t] = v;
}

int fill_doubles(dl_handle* h, double* d, double v, size_t n) {
    if (n == 0) return DL_OK;
    DL_LAUNCH(h, false, fill_kernel<<<(unsigned)((n + 255) / 256), 256, 0, h->stream>>>(d, v, (long long)n));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

}  // namespace dl
