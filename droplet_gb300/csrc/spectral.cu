// spectral.cu -- constant-injection band forcing of the forced-turbulence
// droplet code, externalforce in program/lbm_drop_iht_xy.f90:722-842:
//   u_hat = FFT(u) / N                        (fft_r2c, :894-901)
//   E     = sum_{half spectrum, 1 <= |k| < kc} 0.5 |u_hat|^2 min(2, k3+1)   (:775-795)
//   f_hat = (0.5 eps / E) u_hat on the band, 0 elsewhere                   (:797-818)
//   F     = c2r(f_hat), not normalised         (fft_c2r, :903-908)
// Only the band modes are non-zero, so instead of six full 3-D FFTs per step
// the transform is an exact separable DFT over the 2K+1 (K = kc-1) wavenumbers
// per axis that the band can touch: an x stage over every (y, z) row, then y,
// then z, and the mirror-image synthesis. In the FP64 form every sum runs in
// the same sequential order as the oracle's restatement, so both give the
// same bits; they differ from an FFT by rounding only.
#include "dl_internal.cuh"

#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <vector>

namespace dl {

struct SpArgs {
    int nx, ny, nz, K, kc2;
    const double* u[3];
    double* fo[3];
    const double* twx;
    const double* twy;
    const double* twz;
    double* a1;  // [3][NK][ny][nz] complex -> index ((c*NK + kx)*ny + y)*nz + z
    double* a2;  // [3][NK][NK][nz]
    double* uh;  // [3][NK][NK][K+1]
    double* b1;  // [3][NK][NK][nz]
    double* b2;  // [3][NK][ny][nz]
    DevState* st;
    double half_eps;
    double Nd;
};

// The sums of a wavenumber run over the grid in sequence, so parallelism comes
// from the outputs, and the bound is the FP64 pipe (a warp's FP64 instruction
// takes the SM 16 cycles): k = 0 adds v itself (its twiddle is exactly 1 + 0i),
// table indices advance by k instead of by a division, and the loads of
// several terms are in flight together. Measured at 128^3, kc = 3, before and
// after (us): x stage 317 -> 239, y 117 -> 36, z 70 -> 14, energy 104 -> 6,
// synthesis y 26.5 -> 22, x 289 -> 195.

// m + k in [0, n), |k| < n
__device__ __forceinline__ int step_mod(int m, int k, int n) {
    m += k;
    if (m >= n) m -= n;
    if (m < 0) m += n;
    return m;
}
// k x mod n for |k x| below 2^31
__device__ __forceinline__ int mul_mod(int k, int x, int n) {
    const int m = (k * x) % n;
    return m < 0 ? m + n : m;
}

// x stage: a1[c][kx][y][z] = sum_x u e^{-i 2 pi kx x / nx}. A block takes 32
// rows (one y, 32 z) of a component; its 2K warps take one kx != 0 each, and one
// of them, another in each block, the plain sum of kx = 0 as well. The rows
// come through shared memory, 32 columns at a time, so that the loads run along
// x while every lane sums its own row in order.
__global__ void sp_xstage(const SpArgs a, int nzb) {
    __shared__ double tile[32][33];
    const int NK = 2 * a.K + 1, nw = 2 * a.K;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kx = warp < a.K ? warp - a.K : warp - a.K + 1;
    const bool also0 = (int)(blockIdx.x % nw) == warp;
    const int z0 = (int)(blockIdx.x % nzb) * 32, r = (int)(blockIdx.x / nzb), y = r % a.ny, c = r / a.ny;
    const double* u = a.u[c] + (long long)y * a.nx;
    const double2* tw = reinterpret_cast<const double2*>(a.twx);
    double re = 0.0, im = 0.0, s0 = 0.0;
    int m = 0;
    for (int x0 = 0; x0 < a.nx; x0 += 32) {
        const int w = min(32, a.nx - x0);
        __syncthreads();
        for (int r = warp; r < 32; r += nw)
            if (z0 + r < a.nz && lane < w) tile[r][lane] = __ldg(u + (long long)(z0 + r) * a.ny * a.nx + x0 + lane);
        __syncthreads();
        const double* row = tile[lane];
        int x = 0;
        for (; x + 8 <= w; x += 8) {
            double2 t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                t[k] = __ldg(tw + m);
                m = step_mod(m, kx, a.nx);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const double v = row[x + k];
                re = re + v * t[k].x;
                im = im - v * t[k].y;
            }
        }
        for (; x < w; ++x) {
            const double2 t = __ldg(tw + m);
            re = re + row[x] * t.x;
            im = im - row[x] * t.y;
            m = step_mod(m, kx, a.nx);
        }
        if (also0)
            for (x = 0; x < w; ++x) s0 = s0 + row[x];
    }
    if (z0 + lane >= a.nz) return;
    double2* d = reinterpret_cast<double2*>(a.a1) + ((long long)c * NK * a.ny + y) * a.nz + z0 + lane;
    const long long plane = (long long)a.ny * a.nz;
    d[(kx + a.K) * plane] = make_double2(re, im);
    if (also0) d[a.K * plane] = make_double2(s0, 0.0);
}

// y stage: a2[c][kx][ky][z] = sum_y a1 e^{-i 2 pi ky y / ny}; real and
// imaginary part are two threads' sums (block: 32 z x 2 parts)
__global__ void __launch_bounds__(64) sp_ystage(const SpArgs a) {
    constexpr int B = 16;  // terms in flight
    const int NK = 2 * a.K + 1;
    const int z = blockIdx.x * 32 + (threadIdx.x & 31), part = threadIdx.x >> 5;
    const int kxi = blockIdx.y / NK, kyi = blockIdx.y % NK, c = blockIdx.z;
    if (z >= a.nz) return;
    const int ky = kyi - a.K;
    const double2* v = reinterpret_cast<const double2*>(a.a1) + ((long long)c * NK + kxi) * a.ny * a.nz + z;
    const double2* tw = reinterpret_cast<const double2*>(a.twy);
    double s = 0.0;
    int m = 0;
    for (int y0 = 0; y0 < a.ny; y0 += B) {
        double2 t[B], e[B];
#pragma unroll
        for (int k = 0; k < B; ++k) {
            const int y = min(y0 + k, a.ny - 1);
            t[k] = __ldg(v + (long long)y * a.nz);
            if (ky != 0) e[k] = __ldg(tw + m);
            m = step_mod(m, ky, a.ny);
        }
        if (ky == 0) {
#pragma unroll
            for (int k = 0; k < B; ++k)
                if (y0 + k < a.ny) s = s + (part ? t[k].y : t[k].x);
        } else {
#pragma unroll
            for (int k = 0; k < B; ++k) {
                // re: v0 cos + v1 sin; im: v1 cos - v0 sin
                const double p = part ? t[k].y : t[k].x, q = part ? -t[k].x : t[k].y;
                if (y0 + k < a.ny) s = s + (p * e[k].x + q * e[k].y);
            }
        }
    }
    a.a2[2 * ((((long long)c * NK + kxi) * NK + kyi) * a.nz + z) + part] = s;
}

// z stage: uh[c][kx][ky][kz] = (sum_z a2 e^{-i 2 pi kz z / nz}) / N, kz = 0..K.
// One warp per value: the lanes form the terms of 32 z at once, lane 0 adds the
// real and lane 16 the imaginary ones in order.
__global__ void __launch_bounds__(32) sp_zstage(const SpArgs a) {
    const int lane = threadIdx.x;
    const int kz = blockIdx.x % (a.K + 1), r = blockIdx.x / (a.K + 1);  // r = (c NK + kxi) NK + kyi
    const double2* v = reinterpret_cast<const double2*>(a.a2) + (long long)r * a.nz;
    double s = 0.0;
    for (int z0 = 0; z0 < a.nz; z0 += 32) {
        const int w = min(32, a.nz - z0);
        double pr = 0.0, pi = 0.0;
        if (lane < w) {
            const double2 t = __ldg(v + z0 + lane);
            const double2 e = __ldg(reinterpret_cast<const double2*>(a.twz) + (int)(((long long)kz * (z0 + lane)) % a.nz));
            pr = t.x * e.x + t.y * e.y;
            pi = t.y * e.x - t.x * e.y;
        }
        // (terms past w are +0 and are not added: -0 + 0 would be +0)
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const double tr = __shfl_sync(0xffffffffu, pr, k), ti = __shfl_sync(0xffffffffu, pi, k);
            const double t = lane < 16 ? tr : ti;
            if (k < w) s = s + t;
        }
    }
    if (lane == 0 || lane == 16) a.uh[2 * ((long long)r * (a.K + 1) + kz) + (lane >> 4)] = s / a.Nd;
}

// band energy in the reference's loop order (k3 outer, then k2, then k1, each
// in FFT index order 0 .. K, -K .. -1) and the coefficient 0.5 eps / E: one
// block forms the terms, one thread adds them. MAXT: terms of the largest band
// (K = 4), all of the box 0..K x (2K+1)^2.
constexpr int SP_MAXT = 5 * 9 * 9;
__global__ void __launch_bounds__(256) sp_energy(const SpArgs a) {
    __shared__ double term[SP_MAXT];
    const int NK = 2 * a.K + 1, n = NK * NK * (a.K + 1);
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const int i1 = t % NK, r = t / NK, i2 = r % NK, k3 = r / NK;
        const int k1 = i1 <= a.K ? i1 : i1 - NK, k2 = i2 <= a.K ? i2 : i2 - NK;
        const int kk = k1 * k1 + k2 * k2 + k3 * k3;
        double e[3];
        for (int c = 0; c < 3; ++c) {
            const double* v = a.uh + 2 * ((((long long)c * NK + (k1 + a.K)) * NK + (k2 + a.K)) * (a.K + 1) + k3);
            e[c] = v[0] * v[0] + v[1] * v[1];
        }
        const double w = 2.0 < (double)k3 + 1.0 ? 2.0 : (double)k3 + 1.0;
        // outside the band: +0, which changes no sum of squares
        term[t] = (kk < 1 || kk >= a.kc2) ? 0.0 : 0.5 * (e[0] + e[1] + e[2]) * w;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double energy = 0.0;
    for (int t = 0; t < n; ++t) energy = energy + term[t];
    a.st->sp_energy = energy;
    a.st->sp_coef = a.half_eps / energy;
}

// synthesis, kz then ky then kx, as the c2r of the half spectrum:
// F = sum_kz w(kz) Re(sum f_hat e^{+ik.x}), w = 1 for kz = 0 and 2 otherwise
__global__ void sp_synth_z(const SpArgs a) {
    const int NK = 2 * a.K + 1;
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long total = 3LL * NK * NK * a.nz;
    if (t >= total) return;
    const int z = (int)(t % a.nz);
    long long r = t / a.nz;
    const int kyi = (int)(r % NK);
    r /= NK;
    const int kxi = (int)(r % NK);
    const int c = (int)(r / NK);
    const int kx = kxi - a.K, ky = kyi - a.K;
    const double coef = a.st->sp_coef;
    double re = 0.0, im = 0.0;
    for (int kz = 0; kz <= a.K; ++kz) {
        const int kk = kx * kx + ky * ky + kz * kz;
        if (kk < 1 || kk >= a.kc2) continue;
        const double* v = a.uh + 2 * ((((long long)c * NK + kxi) * NK + kyi) * (a.K + 1) + kz);
        const double fre = coef * v[0], fim = coef * v[1];
        const double w = kz == 0 ? 1.0 : 2.0;
        const int m = (int)(((long long)kz * z) % a.nz);
        const double cz_ = a.twz[2 * m], sz_ = a.twz[2 * m + 1];
        re = re + w * (fre * cz_ - fim * sz_);
        im = im + w * (fre * sz_ + fim * cz_);
    }
    double* d = a.b1 + 2 * ((((long long)c * NK + kxi) * NK + kyi) * a.nz + z);
    d[0] = re;
    d[1] = im;
}

__global__ void sp_synth_y(const SpArgs a) {
    const int NK = 2 * a.K + 1;
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long total = 3LL * NK * a.ny * a.nz;
    if (t >= total) return;
    const int z = (int)(t % a.nz);
    long long r = t / a.nz;
    const int y = (int)(r % a.ny);
    r /= a.ny;
    const int kxi = (int)(r % NK);
    const int c = (int)(r / NK);
    const double2* b1 = reinterpret_cast<const double2*>(a.b1) + ((long long)c * NK + kxi) * NK * a.nz + z;
    double re = 0.0, im = 0.0;
    int m = mul_mod(-a.K, y, a.ny);
    for (int kyi = 0; kyi < NK; ++kyi) {
        const double2 v = __ldg(b1 + (long long)kyi * a.nz);
        if (kyi == a.K) {
            re = re + v.x;
            im = im + v.y;
        } else {
            const double2 e = __ldg(reinterpret_cast<const double2*>(a.twy) + m);
            re = re + (v.x * e.x - v.y * e.y);
            im = im + (v.x * e.y + v.y * e.x);
        }
        m = step_mod(m, y, a.ny);
    }
    reinterpret_cast<double2*>(a.b2)[(((long long)c * NK + kxi) * a.ny + y) * a.nz + z] = make_double2(re, im);
}

// a warp's 32 sites along x share their row's coefficients; a thread takes the
// three components of its site (block: 32 x by 4 rows of the flattened y, z)
template <int K>
__global__ void __launch_bounds__(128) sp_synth_x(const SpArgs a, int nxb) {
    constexpr int NK = 2 * K + 1;
    const int x = (int)(blockIdx.x % nxb) * 32 + (threadIdx.x & 31);
    const long long r = (long long)(blockIdx.x / nxb) * 4 + (threadIdx.x >> 5);
    const int z = (int)(r / a.ny), y = (int)(r - (long long)z * a.ny);
    if (x >= a.nx || z >= a.nz) return;
    const double2* b2 = reinterpret_cast<const double2*>(a.b2) + (long long)y * a.nz + z;
    const long long plane = (long long)a.ny * a.nz;
    double2 e[NK];
    int m = mul_mod(-K, x, a.nx);
#pragma unroll
    for (int k = 0; k < NK; ++k) {
        if (k != K) e[k] = __ldg(reinterpret_cast<const double2*>(a.twx) + m);
        m = step_mod(m, x, a.nx);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double2 v[NK];
#pragma unroll
        for (int k = 0; k < NK; ++k) v[k] = __ldg(b2 + (c * NK + k) * plane);
        double f = v[0].x * e[0].x - v[0].y * e[0].y;
#pragma unroll
        for (int k = 1; k < NK; ++k) f = k == K ? f + v[k].x : f + (v[k].x * e[k].x - v[k].y * e[k].y);
        a.fo[c][r * a.nx + x] = f;
    }
}

static void launch_synth_x(const SpArgs& a, cudaStream_t s) {
    const int nxb = (a.nx + 31) / 32;
    const unsigned g = (unsigned)(nxb * (((long long)a.ny * a.nz + 3) / 4));
    if (a.K == 1) sp_synth_x<1><<<g, 128, 0, s>>>(a, nxb);
    else if (a.K == 2) sp_synth_x<2><<<g, 128, 0, s>>>(a, nxb);
    else if (a.K == 3) sp_synth_x<3><<<g, 128, 0, s>>>(a, nxb);
    else sp_synth_x<4><<<g, 128, 0, s>>>(a, nxb);
}

// FP32 forms: the x stage with one warp per (y, z) row (lanes over x, FP32
// sums, reduced across the warp), and the x synthesis writing FP32 forces.
// The small y / z stages and the energy are shared with the FP64 form.
constexpr int SP_KMAX = 4;  // supports kc <= 5

__global__ void sp_xstage_f32(const float* __restrict__ u1, const float* __restrict__ u2,
                              const float* __restrict__ u3, double* __restrict__ a1, int nx, int ny, int nz, int K,
                              const float* __restrict__ tw) {
    const int lane = threadIdx.x & 31;
    const long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    if (row >= (long long)ny * nz) return;
    const int z = (int)(row / ny), y = (int)(row - (long long)z * ny);
    const int NK = 2 * K + 1;
    const float* u[3] = {u1, u2, u3};
    const long long base = ((long long)z * ny + y) * nx;
    float re[3][2 * SP_KMAX + 1], im[3][2 * SP_KMAX + 1];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        for (int k = 0; k < NK; ++k) re[c][k] = im[c][k] = 0.f;
    for (int x = lane; x < nx; x += 32) {
        const float v[3] = {u[0][base + x], u[1][base + x], u[2][base + x]};
        for (int k = 0; k < NK; ++k) {
            int m = ((k - K) * x) % nx;
            m = m < 0 ? m + nx : m;
            const float cs = tw[2 * m], sn = tw[2 * m + 1];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                re[c][k] += v[c] * cs;
                im[c][k] -= v[c] * sn;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
        for (int k = 0; k < NK; ++k) {
            float r = re[c][k], i = im[c][k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                r += __shfl_xor_sync(0xffffffffu, r, o);
                i += __shfl_xor_sync(0xffffffffu, i, o);
            }
            if (lane == 0) {
                double* d = a1 + 2 * ((((long long)c * NK + k) * ny + y) * nz + z);
                d[0] = (double)r;
                d[1] = (double)i;
            }
        }
}

__global__ void sp_synth_x_f32(const double* __restrict__ b2, float* __restrict__ fx, float* __restrict__ fy,
                               float* __restrict__ fz, int nx, int ny, int nz, int K, const float* __restrict__ tw) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long N = (long long)nx * ny * nz;
    if (s >= N) return;
    const int x = (int)(s % nx);
    const long long r = s / nx;
    const int y = (int)(r % ny), z = (int)(r / ny);
    const int NK = 2 * K + 1;
    float out[3] = {0.f, 0.f, 0.f};
    for (int k = 0; k < NK; ++k) {
        int m = ((k - K) * x) % nx;
        m = m < 0 ? m + nx : m;
        const float cs = tw[2 * m], sn = tw[2 * m + 1];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double* v = b2 + 2 * ((((long long)c * NK + k) * ny + y) * nz + z);
            out[c] += (float)v[0] * cs - (float)v[1] * sn;
        }
    }
    fx[s] = out[0];
    fy[s] = out[1];
    fz[s] = out[2];
}

// ---- adjoint of the band force (reverse pass of a step with the spectral force) ----
// F = coef v with v = P u, the band-pass of u (sum over the band of w Re(u_hat
// e^{ik.x}), u_hat = DFT(u)/N), coef = 0.5 eps / E and E = sum w 0.5 |u_hat|^2 =
// |v|^2 / 2N. For lF = dL/dF, since P is a symmetric projection and dE/du = v/N:
//   dL/du = coef P lF - (s coef / (E N)) v,   s = sum_x lF . v = N sum w Re(u_hat conj(L_hat)),
// with L_hat the band coefficients of lF: one synthesis of the combined
// coefficients coef L_hat - (s coef / (E N)) u_hat. One block; reads E and coef
// that sp_energy left, writes the combination into uh and sets coef = 1 for
// the synthesis kernels.
__global__ void sp_adj_combine(const SpArgs a, const double* __restrict__ lh) {
    __shared__ double s_part[32];
    const int NK = 2 * a.K + 1;
    const int nv = 3 * NK * NK * (a.K + 1);
    const double E = a.st->sp_energy, coef = a.st->sp_coef;
    double s = 0.0;
    for (int t = threadIdx.x; t < nv; t += blockDim.x) {
        const int kz = t % (a.K + 1), r = t / (a.K + 1), kyi = r % NK, kxi = (r / NK) % NK;
        const int kx = kxi - a.K, ky = kyi - a.K, kk = kx * kx + ky * ky + kz * kz;
        if (kk < 1 || kk >= a.kc2) continue;
        const double w = kz == 0 ? 1.0 : 2.0;
        s += w * (a.uh[2 * t] * lh[2 * t] + a.uh[2 * t + 1] * lh[2 * t + 1]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = s;
    __syncthreads();
    double tot = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += s_part[w];
    const double g = tot * coef / E;  // s coef / (E N), s = N tot
    for (int t = threadIdx.x; t < 2 * nv; t += blockDim.x) a.uh[t] = coef * lh[t] - g * a.uh[t];
    __syncthreads();
    if (threadIdx.x == 0) a.st->sp_coef = 1.0;
}

// the x synthesis added into FP32 arrays
__global__ void sp_synth_x_add_f32(const double* __restrict__ b2, float* __restrict__ o1, float* __restrict__ o2,
                                   float* __restrict__ o3, int nx, int ny, int nz, int K,
                                   const float* __restrict__ tw) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long N = (long long)nx * ny * nz;
    if (s >= N) return;
    const int x = (int)(s % nx);
    const long long r = s / nx;
    const int y = (int)(r % ny), z = (int)(r / ny);
    const int NK = 2 * K + 1;
    float out[3] = {0.f, 0.f, 0.f};
    for (int k = 0; k < NK; ++k) {
        int m = ((k - K) * x) % nx;
        m = m < 0 ? m + nx : m;
        const float cs = tw[2 * m], sn = tw[2 * m + 1];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double* v = b2 + 2 * ((((long long)c * NK + k) * ny + y) * nz + z);
            out[c] += (float)v[0] * cs - (float)v[1] * sn;
        }
    }
    o1[s] += out[0];
    o2[s] += out[1];
    o3[s] += out[2];
}

static int upload_twiddle(dl_handle* h, int n, double** d) {
    std::vector<double> t(2 * (size_t)n);
    const double pi = acos(-1.0);
    for (int m = 0; m < n; ++m) {
        const double ang = 2.0 * pi * (double)m / (double)n;
        t[2 * m] = cos(ang);
        t[2 * m + 1] = sin(ang);
    }
    DL_CUDA(h, cudaMalloc(d, sizeof(double) * 2 * n));
    DL_CUDA(h, cudaMemcpy(*d, t.data(), sizeof(double) * 2 * n, cudaMemcpyHostToDevice));
    return DL_OK;
}

int spectral_alloc(dl_handle* h) {
    SpectralPlan& sp = h->sp;
    memset(&sp, 0, sizeof(sp));
    const int K = h->P.kc - 1;
    sp.K = K;
    if (K < 1) return DL_OK;
    if (2 * K + 1 > h->nx || 2 * K + 1 > h->ny || K + 1 > h->nz / 2) {
        // no band plan: dl_set_force(DL_FORCE_SPECTRAL) refuses; the step itself works
        sp.K = 0;
        return DL_OK;
    }
    const int NK = 2 * K + 1;
    int rc;
    if ((rc = upload_twiddle(h, h->nx, &sp.d_twx)) != DL_OK) return rc;
    if ((rc = upload_twiddle(h, h->ny, &sp.d_twy)) != DL_OK) return rc;
    if ((rc = upload_twiddle(h, h->nz, &sp.d_twz)) != DL_OK) return rc;
    if (K > SP_KMAX) return set_error(h, DL_ERR_ARG, "kc=%d above the supported maximum %d", h->P.kc, SP_KMAX + 1);
    {
        std::vector<float> t(2 * (size_t)h->nx);
        const double pi = acos(-1.0);
        for (int m = 0; m < h->nx; ++m) {
            t[2 * m] = (float)cos(2.0 * pi * m / h->nx);
            t[2 * m + 1] = (float)sin(2.0 * pi * m / h->nx);
        }
        DL_CUDA(h, cudaMalloc(&sp.d_twxf, sizeof(float) * 2 * h->nx));
        DL_CUDA(h, cudaMemcpy(sp.d_twxf, t.data(), sizeof(float) * 2 * h->nx, cudaMemcpyHostToDevice));
    }
    const size_t rows = (size_t)h->ny * h->nz;
    DL_CUDA(h, cudaMalloc(&sp.d_a1, sizeof(double) * 2 * 3 * NK * rows));
    DL_CUDA(h, cudaMalloc(&sp.d_b2, sizeof(double) * 2 * 3 * NK * rows));
    // a2 and b1 share one buffer: [3][NK][NK][nz] complex each
    DL_CUDA(h, cudaMalloc(&sp.d_uh, sizeof(double) * 2 * 3 * NK * NK * ((size_t)K + 1 + 2 * (size_t)h->nz)));
    int nm = 0;
    for (int kz = 0; kz <= K; ++kz)
        for (int ky = -K; ky <= K; ++ky)
            for (int kx = -K; kx <= K; ++kx) {
                int kk = kx * kx + ky * ky + kz * kz;
                if (kk >= 1 && kk < h->P.kc * h->P.kc) ++nm;
            }
    sp.nmodes = nm;
    return DL_OK;
}

void spectral_free(dl_handle* h) {
    SpectralPlan& sp = h->sp;
    cudaFree(sp.d_twx);
    cudaFree(sp.d_twy);
    cudaFree(sp.d_twz);
    cudaFree(sp.d_a1);
    cudaFree(sp.d_b2);
    cudaFree(sp.d_uh);
    cudaFree(sp.d_twxf);
    cudaFree(sp.d_lh);
    memset(&sp, 0, sizeof(sp));
}

static void fill_sp(dl_handle* h, SpArgs& a) {
    memset(&a, 0, sizeof(a));
    const SpectralPlan& sp = h->sp;
    const int NK = 2 * sp.K + 1;
    a.nx = h->nx;
    a.ny = h->ny;
    a.nz = h->nz;
    a.K = sp.K;
    a.kc2 = h->P.kc * h->P.kc;
    a.twx = sp.d_twx;
    a.twy = sp.d_twy;
    a.twz = sp.d_twz;
    a.a1 = sp.d_a1;
    a.b2 = sp.d_b2;
    a.uh = sp.d_uh;
    a.a2 = sp.d_uh + 2 * 3 * NK * NK * (size_t)(sp.K + 1);
    a.b1 = a.a2 + 2 * 3 * NK * NK * (size_t)h->nz;
    a.st = h->d_state;
    a.half_eps = 0.5 * h->P.eps;
    a.Nd = (double)h->nx * (double)h->ny * (double)h->nz;
}

static inline unsigned nb(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

int spectral_force_fp64(dl_handle* h, const double* u1, const double* u2, const double* u3, double* fx,
                        double* fy, double* fz) {
    SpArgs a;
    fill_sp(h, a);
    a.u[0] = u1;
    a.u[1] = u2;
    a.u[2] = u3;
    a.fo[0] = fx;
    a.fo[1] = fy;
    a.fo[2] = fz;
    const int NK = 2 * a.K + 1;
    cudaStream_t s = h->stream;
    DL_LAUNCH(h, false, (sp_xstage<<<(unsigned)((h->nz + 31) / 32 * 3LL * h->ny), 64 * a.K, 0, s>>>(a, (h->nz + 31) / 32)));
    DL_LAUNCH(h, false, (sp_ystage<<<dim3((h->nz + 31) / 32, NK * NK, 3), 64, 0, s>>>(a)));
    DL_LAUNCH(h, false, (sp_zstage<<<3 * NK * NK * (a.K + 1), 32, 0, s>>>(a)));
    DL_LAUNCH(h, false, (sp_energy<<<1, 256, 0, s>>>(a)));
    DL_LAUNCH(h, false, sp_synth_z<<<nb(3LL * NK * NK * h->nz, 128), 128, 0, s>>>(a));
    DL_LAUNCH(h, false, sp_synth_y<<<nb(3LL * NK * h->ny * h->nz, 128), 128, 0, s>>>(a));
    DL_LAUNCH(h, false, launch_synth_x(a, s));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

// forward part only: sp.d_uh = band coefficients u_hat / N of an FP32 u
int spectral_project_f32(dl_handle* h, const float* u1, const float* u2, const float* u3) {
    SpArgs a;
    fill_sp(h, a);
    const int NK = 2 * a.K + 1;
    cudaStream_t s = h->stream;
    const long long rows = (long long)h->ny * h->nz;
    DL_LAUNCH(h, false, sp_xstage_f32<<<nb(rows * 32, 256), 256, 0, s>>>(u1, u2, u3, a.a1, h->nx, h->ny, h->nz, a.K,
                                                                        h->sp.d_twxf));
    DL_LAUNCH(h, false, (sp_ystage<<<dim3((h->nz + 31) / 32, NK * NK, 3), 64, 0, s>>>(a)));
    DL_LAUNCH(h, false, (sp_zstage<<<3 * NK * NK * (a.K + 1), 32, 0, s>>>(a)));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

// dL/du of the band force added into lu, from dL/dF (lf) and the u the force was
// computed from
int spectral_adjoint_f32(dl_handle* h, const float* lf1, const float* lf2, const float* lf3, const float* u1,
                         const float* u2, const float* u3, float* lu1, float* lu2, float* lu3) {
    SpectralPlan& sp = h->sp;
    if (sp.K < 1) return set_error(h, DL_ERR_STATE, "no band plan for the spectral force");
    const int NK = 2 * sp.K + 1;
    const size_t nuh = (size_t)2 * 3 * NK * NK * (sp.K + 1);
    if (!sp.d_lh) DL_CUDA(h, cudaMalloc(&sp.d_lh, sizeof(double) * nuh));
    int rc = spectral_project_f32(h, lf1, lf2, lf3);
    if (rc != DL_OK) return rc;
    DL_CUDA(h, cudaMemcpyAsync(sp.d_lh, sp.d_uh, sizeof(double) * nuh, cudaMemcpyDeviceToDevice, h->stream));
    rc = spectral_project_f32(h, u1, u2, u3);
    if (rc != DL_OK) return rc;
    SpArgs a;
    fill_sp(h, a);
    cudaStream_t s = h->stream;
    const long long N = (long long)h->N;
    DL_LAUNCH(h, false, (sp_energy<<<1, 256, 0, s>>>(a)));
    DL_LAUNCH(h, false, sp_adj_combine<<<1, 256, 0, s>>>(a, sp.d_lh));
    DL_LAUNCH(h, false, sp_synth_z<<<nb(3LL * NK * NK * h->nz, 128), 128, 0, s>>>(a));
    DL_LAUNCH(h, false, sp_synth_y<<<nb(3LL * NK * h->ny * h->nz, 128), 128, 0, s>>>(a));
    DL_LAUNCH(h, false, sp_synth_x_add_f32<<<nb(N, 256), 256, 0, s>>>(a.b2, lu1, lu2, lu3, h->nx, h->ny, h->nz, a.K,
                                                                       sp.d_twxf));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

int spectral_force_f32(dl_handle* h, const float* u1, const float* u2, const float* u3, float* fx, float* fy,
                       float* fz) {
    SpArgs a;
    fill_sp(h, a);
    const int NK = 2 * a.K + 1;
    const long long N = (long long)h->N;
    cudaStream_t s = h->stream;
    const long long rows = (long long)h->ny * h->nz;
    DL_LAUNCH(h, false, sp_xstage_f32<<<nb(rows * 32, 256), 256, 0, s>>>(u1, u2, u3, a.a1, h->nx, h->ny, h->nz, a.K,
                                                                        h->sp.d_twxf));
    DL_LAUNCH(h, false, (sp_ystage<<<dim3((h->nz + 31) / 32, NK * NK, 3), 64, 0, s>>>(a)));
    DL_LAUNCH(h, false, (sp_zstage<<<3 * NK * NK * (a.K + 1), 32, 0, s>>>(a)));
    DL_LAUNCH(h, false, (sp_energy<<<1, 256, 0, s>>>(a)));
    DL_LAUNCH(h, false, sp_synth_z<<<nb(3LL * NK * NK * h->nz, 128), 128, 0, s>>>(a));
    DL_LAUNCH(h, false, sp_synth_y<<<nb(3LL * NK * h->ny * h->nz, 128), 128, 0, s>>>(a));
    DL_LAUNCH(h, false, sp_synth_x_f32<<<nb(N, 256), 256, 0, s>>>(a.b2, fx, fy, fz, h->nx, h->ny, h->nz, a.K,
                                                                   h->sp.d_twxf));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

}  // namespace dl
