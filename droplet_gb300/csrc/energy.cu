// energy.cu -- in-situ turbulence and free-energy diagnostics of the current
// fields (dl_energy):
//  * the shell-binned kinetic-energy spectrum of enesupe_cal,
//    program/turbulence_hit_xy.f90:588-645: u_hat = FFT(u)/N (fft_r2c,
//    :725-730), summed over the reference's index set k1 in [0,nx),
//    k2 in [0,ny), k3 in [0,nz/2] with weight 1 on k3 = 0 and 2 elsewhere,
//    into bin int(|k|) + 1 with the signed wavenumbers of the function judge (:739-746);
//    the FFTs are cuFFT D2Z transforms in FP64, modes outside the stored half
//    are read through Hermitian symmetry;
//  * sums of the bulk free energy psi = phi T ln(phi/(1 - b phi)) - a phi^2
//    (free_energy_cal, program/energy_budget.f90:1012-1023), of the chemical
//    potential mu = T ln(phi/(1 - b phi)) + T/(1 - b phi) - 2 a phi
//    - kappag lap(phi) (chemical_potencial_cal, :998-1010; the 14-neighbour
//    Laplacian of various_cal) and of |grad phi|^2.
#include "dl_internal.cuh"
#include "diag_site.cuh"

#include <cufft.h>
#include <math.h>
#include <string.h>
#include <vector>

namespace dl {

constexpr int EN_THREADS = 256;
constexpr int EN_BLOCKS = 608;  // 4 x 152 SMs
constexpr int EN_BIN_BLOCKS = 304;
constexpr int EN_SMEM_BINS = 2048;  // bins histogrammed in shared memory first

// one velocity component as doubles (the FFT input)
__global__ void en_component(const void* mac, int fast, int c, long long N, double* __restrict__ out) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= N) return;
    out[s] = fast ? (double)((const float*)mac)[(c + 1) * N + s] : ((const double*)mac)[(c + 1) * N + s];
}

// acc += |u_hat|^2 / N^2 over the stored half spectrum
__global__ void en_accumulate(const cufftDoubleComplex* __restrict__ uh, long long M, double invN2, int first,
                              double* __restrict__ acc) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= M) return;
    const double v = (uh[t].x * uh[t].x + uh[t].y * uh[t].y) * invN2;
    acc[t] = first ? v : acc[t] + v;
}

__device__ __forceinline__ int en_signed(int k, int n) { return k >= n / 2 + 1 ? k - n : k; }

// spectrum[int(|k|)] += 0.5 |u_hat|^2 w over the reference's index set
__global__ void __launch_bounds__(EN_THREADS) en_bin(const double* __restrict__ acc, int nx, int ny, int nz,
                                                    int nbins, double* __restrict__ spectrum) {
    __shared__ double hist[EN_SMEM_BINS];
    const int nsh = nbins < EN_SMEM_BINS ? nbins : EN_SMEM_BINS;
    for (int b = threadIdx.x; b < nsh; b += blockDim.x) hist[b] = 0.0;
    __syncthreads();
    const int nxh = nx / 2 + 1;
    const long long total = (long long)nx * ny * (nz / 2 + 1);
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int k1 = (int)(t % nx);
        const long long r = t / nx;
        const int k2 = (int)(r % ny);
        const int k3 = (int)(r / ny);
        // stored index [iz][iy][ix] of (k1, k2, k3) or of its partner -k
        int ix = k1, iy = k2, iz = k3;
        if (k1 >= nxh) {
            ix = nx - k1;
            iy = (ny - k2) % ny;
            iz = (nz - k3) % nz;
        }
        const double e2 = acc[((long long)iz * ny + iy) * nxh + ix];
        const int s1 = en_signed(k1, nx), s2 = en_signed(k2, ny), s3 = en_signed(k3, nz);
        const int kidx = (int)sqrt((double)(s1 * s1 + s2 * s2 + s3 * s3));  // bin index - 1
        if (kidx >= nbins) continue;
        const double v = 0.5 * e2 * (k3 == 0 ? 1.0 : 2.0);
        if (kidx < nsh) atomicAdd(hist + kidx, v);
        else atomicAdd(spectrum + kidx, v);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nsh; b += blockDim.x)
        if (hist[b] != 0.0) atomicAdd(spectrum + b, hist[b]);
}

// per-block partial sums of psi, mu and |grad phi|^2
struct EnArgs {
    int nx, ny, nz, ltx, chunk;  // ltx, chunk: as in diag_site.cuh
    long long N;
    const void* mac;
    double phi_off, T, a, b, kappag, inv_lap, inv_grad;
    double* part;  // [EN_BLOCKS][3]
};

// A block takes 32 x 8 column tiles, `chunk` planes at a time, and marches them
// with four planes of phi - phi_off (tile and one-cell ring, as doubles) in
// shared memory, so that a value is converted once and not at each of its 15
// readers. The FP64 pipe is the bound: the seven opposite pairs give the sums
// of the Laplacian and the differences of the gradient (31 additions; sums over
// the 14 neighbours with products by c took 113), one reciprocal serves both
// quotients, the stencil factors are applied to the sums. 128^3 FP32: 640 ->
// 346 us, a third of it the logarithm.
static_assert(EN_THREADS == DIAG_NT, "the tiles of diag_site.cuh");
template <typename T>
__global__ void __launch_bounds__(EN_THREADS) en_free_energy(const EnArgs a) {
    __shared__ double ring[4][DIAG_P];
    const T* __restrict__ phi = (const T*)a.mac;
    const int TX = 1 << a.ltx, TY = EN_THREADS >> a.ltx, EX = TX + 2, np = EX * (TY + 2);
    const int tid = threadIdx.x, tx = tid & (TX - 1), ty = tid >> a.ltx;
    const int gx = (a.nx + TX - 1) / TX, gy = (a.ny + TY - 1) / TY, gz = (a.nz + a.chunk - 1) / a.chunk;
    const long long nxy = (long long)a.nx * a.ny, items = (long long)gx * gy * gz;
    const int k0 = (ty + 1) * EX + tx + 1;
    double psi = 0.0, mu = 0.0, lap = 0.0, grad = 0.0;
    for (long long it = blockIdx.x; it < items; it += gridDim.x) {
        const int bz = (int)(it / (gx * gy)), r = (int)(it - (long long)bz * gx * gy), by = r / gx, bx = r - by * gx;
        const int x0 = bx * TX, y0 = by * TY, z0 = bz * a.chunk, z1 = min(z0 + a.chunk, a.nz);
        long long off[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int p = tid + j * EN_THREADS, ey = p / EX, ex = p - ey * EX;
            const int x = (x0 - 1 + ex + a.nx) % a.nx, y = (y0 - 1 + ey + a.ny) % a.ny;
            off[j] = x + (long long)a.nx * y;
        }
        auto load = [&](int z) {
            const long long zo = nxy * (z < 0 ? z + a.nz : (z >= a.nz ? z - a.nz : z));
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (tid + j * EN_THREADS < np) ring[z & 3][tid + j * EN_THREADS] = (double)__ldg(phi + zo + off[j]);
        };
        const bool act = x0 + tx < a.nx && y0 + ty < a.ny;
        __syncthreads();  // the previous item's readers
        load(z0 - 1);
        load(z0);
        load(z0 + 1);
        for (int z = z0; z < z1; ++z) {
            __syncthreads();
            if (z + 1 < z1) load(z + 2);
            const double *m = ring[(z - 1) & 3] + k0, *c = ring[z & 3] + k0, *p = ring[(z + 1) & 3] + k0;
            if (!act) continue;
            double s = 0.0, d[7];
            auto pair = [&](int k, double vp, double vm) {
                s = k ? s + (vp + vm) : vp + vm;
                d[k] = vp - vm;
            };
            pair(0, c[1], c[-1]);
            pair(1, c[EX], c[-EX]);
            pair(2, p[0], m[0]);
            pair(3, p[EX + 1], m[-EX - 1]);   // c_7 = (+,+,+)
            pair(4, p[EX - 1], m[-EX + 1]);   // c_8 = (-,+,+)
            pair(5, p[-EX + 1], m[EX - 1]);   // c_9 = (+,-,+)
            pair(6, m[EX + 1], p[-EX - 1]);   // c_10 = (+,+,-)
            const double v = c[0], ph = a.phi_off + v;
            lap += __fma_rn(-14.0, v, s);
            const double e = d[3] + d[4], f = d[5] + d[6], g = d[3] - d[4], h = d[5] - d[6];
            const double g0 = d[0] + (g + f), g1 = d[1] + (e - h), g2 = d[2] + (e + h);
            grad = __fma_rn(g0, g0, grad);
            grad = __fma_rn(g1, g1, grad);
            grad = __fma_rn(g2, g2, grad);
            const double rec = 1.0 / __fma_rn(-a.b, ph, 1.0);
            const double tl = a.T * log(ph * rec), aph = a.a * ph;
            psi += ph * (tl - aph);
            mu += __fma_rn(-2.0, aph, __fma_rn(a.T, rec, tl));
        }
    }
    const double acc[3] = {psi, __fma_rn(-a.kappag * a.inv_lap, lap, mu), grad * a.inv_grad * a.inv_grad};
    __shared__ double sh[EN_THREADS / 32][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) sh[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0;
        for (int w = 0; w < EN_THREADS / 32; ++w) v += sh[w][threadIdx.x];
        a.part[blockIdx.x * 3 + threadIdx.x] = v;
    }
}

void energy_free(dl_handle* h) {
    if (h->en_plan_ok) cufftDestroy((cufftHandle)h->en_plan);
    h->en_plan_ok = 0;
    cudaFree(h->en_buf);
    h->en_buf = nullptr;
}

// enqueues the spectrum; its bins are left on the device
static int en_spectrum(dl_handle* h, long long nbins, double** d_bins) {
    const int nx = h->nx, ny = h->ny, nz = h->nz;
    const long long N = (long long)h->N;
    const long long M = (long long)nz * ny * (nx / 2 + 1);  // stored half spectrum
    // buffer: input N doubles | output M complex | acc M doubles | bins
    double* in = h->en_buf;
    cufftDoubleComplex* out = (cufftDoubleComplex*)(in + N + (N & 1));
    double* acc = (double*)(out + M);
    double* bins = acc + M;
    if (!h->en_plan_ok) {
        cufftHandle plan;
        if (cufftPlan3d(&plan, nz, ny, nx, CUFFT_D2Z) != CUFFT_SUCCESS)
            return set_error(h, DL_ERR_CUDA, "cufftPlan3d(D2Z) failed");
        h->en_plan = (long long)plan;
        h->en_plan_ok = 1;
    }
    const cufftHandle plan = (cufftHandle)h->en_plan;
    if (cufftSetStream(plan, h->stream) != CUFFT_SUCCESS) return set_error(h, DL_ERR_CUDA, "cufftSetStream failed");
    const bool fast = h->form != DL_FORM_FP64;
    const void* mac = fast ? (const void*)h->mac32[h->cur] : (const void*)h->mac64[h->cur];
    const double invN2 = 1.0 / ((double)N * (double)N);
    for (int c = 0; c < 3; ++c) {
        DL_LAUNCH(h, false, (en_component<<<(unsigned)((N + 255) / 256), 256, 0, h->stream>>>(mac, fast, c, N, in)));
        if (cufftExecD2Z(plan, in, out) != CUFFT_SUCCESS) return set_error(h, DL_ERR_CUDA, "cufftExecD2Z failed");
        DL_LAUNCH(h, false,
                  (en_accumulate<<<(unsigned)((M + 255) / 256), 256, 0, h->stream>>>(out, M, invN2, c == 0, acc)));
    }
    DL_CUDA(h, cudaMemsetAsync(bins, 0, sizeof(double) * (size_t)nbins, h->stream));
    DL_LAUNCH(h, false, (en_bin<<<EN_BIN_BLOCKS, EN_THREADS, 0, h->stream>>>(acc, nx, ny, nz, (int)nbins, bins)));
    DL_CUDA(h, cudaGetLastError());
    *d_bins = bins;
    return DL_OK;
}

int energy_diagnostics(dl_handle* h, dl_energy_diag* out, double* spectrum_host, long long nbins) {
    if (nbins < 0 || (nbins > 0 && !spectrum_host)) return set_error(h, DL_ERR_ARG, "bad spectrum buffer");
    const long long N = (long long)h->N;
    const long long M = (long long)h->nz * h->ny * (h->nx / 2 + 1);
    const size_t need = sizeof(double) * (size_t)(N + 1 + 2 * M + M + (nbins > 0 ? nbins : 0) + 3 * EN_BLOCKS);
    if (need > h->en_bytes) {
        cudaFree(h->en_buf);
        h->en_buf = nullptr;
        h->en_bytes = 0;
        DL_CUDA(h, cudaMalloc(&h->en_buf, need));
        h->en_bytes = need;
    }
    memset(out, 0, sizeof(*out));
    // free-energy sums (partials at the end of the buffer)
    EnArgs a;
    memset(&a, 0, sizeof(a));
    a.nx = h->nx;
    a.ny = h->ny;
    a.nz = h->nz;
    a.N = N;
    const bool fast = h->form != DL_FORM_FP64;
    a.mac = fast ? (const void*)h->mac32[h->cur] : (const void*)h->mac64[h->cur];
    a.phi_off = fast ? h->P.phi1 : 0.0;
    a.T = h->P.T;
    a.a = h->P.a;
    a.b = h->P.b;
    a.kappag = h->P.kappag;
    a.inv_lap = 1.0 / (5.0 * h->P.ds * h->P.ds);
    a.inv_grad = 1.0 / (10.0 * h->P.ds);
    a.part = h->en_buf + h->en_bytes / sizeof(double) - 3 * EN_BLOCKS;
    a.ltx = diag_tile(a.nx, a.ny);
    a.chunk = diag_chunk(diag_tiles(a.nx, a.ny, a.ltx), a.nz, EN_BLOCKS, 0.7);
    if (fast) DL_LAUNCH(h, false, (en_free_energy<float><<<EN_BLOCKS, EN_THREADS, 0, h->stream>>>(a)));
    else DL_LAUNCH(h, false, (en_free_energy<double><<<EN_BLOCKS, EN_THREADS, 0, h->stream>>>(a)));
    DL_CUDA(h, cudaGetLastError());
    double* d_bins = nullptr;
    if (nbins > 0) {
        const int rc = en_spectrum(h, nbins, &d_bins);
        if (rc != DL_OK) return rc;
    }
    // everything is enqueued before the first copy waits for it
    std::vector<double> part(3 * EN_BLOCKS);
    DL_CUDA(h, cudaMemcpyAsync(part.data(), a.part, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, h->stream));
    if (nbins > 0)
        DL_CUDA(h, cudaMemcpyAsync(spectrum_host, d_bins, sizeof(double) * (size_t)nbins, cudaMemcpyDeviceToHost,
                                   h->stream));
    DL_CUDA(h, cudaStreamSynchronize(h->stream));
    double sums[3] = {0.0, 0.0, 0.0};
    for (int b = 0; b < EN_BLOCKS; ++b)
        for (int k = 0; k < 3; ++k) sums[k] += part[3 * b + k];
    out->psi_sum = sums[0];
    out->mu_sum = sums[1];
    out->grad_sq_sum = sums[2];
    out->nbins = nbins;
    for (long long b = 0; b < nbins; ++b) out->spectrum_sum += spectrum_host[b];
    out->step = h->step;
    return DL_OK;
}

}  // namespace dl
