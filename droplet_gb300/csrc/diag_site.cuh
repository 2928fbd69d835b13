// diag_site.cuh -- the per-site terms of the whole-domain diagnostics that
// dl_reduce and dl_reduce_static sum (one definition for both):
// conservation sums (phi, p, momentum), kinetic energy, dissipation
// 2 nu(phi) S:S with the reference's 14-neighbour gradient stencil
// (program/lbm_drop_xy.f90:615-633; dissipation convention of
// program/energy_budget.f90:1494), droplet volume (phi above the mid value,
// threshold of program/percolation.f90:112), pressure inside and outside,
// and the moments of w = (phi - phi1)/(phi2 - phi1) for the deformation D
// (prototype_program/two-phase/drop8_mpi.f90:812-970), FP64 throughout.
//
// The stencil weights are -1, 0, +1, so the gradient is formed by signed
// additions only (a product with a zero weight is never issued); it and the
// strain contraction S:S (over the six distinct entries of the symmetric
// strain) are formed in the storage type of the fields (FP32 for the FP32 and
// FP16 forms, as their step forms the LES strain; FP64 for the FP64 form),
// then scaled by 1/(4 graddiv^2) in FP64: GB300's FP64 pipe is narrow.
#pragma once

#include "dl_internal.cuh"
#include "dl_device.cuh"

namespace dl {

constexpr int DIAG_NSUM = 24;  // sums; then min and max of phi

struct DiagConsts {
    int nx, ny, nz;
    long long N;
    double phi1, phi_off, p_off;  // stored phi and p are phi - phi_off, p - p_off
    double inv_span, mid, nu1, dnu;
    double sfac;  // 1 / (4 graddiv^2)
    int ltx, chunk;  // diag_march
};

// Blocks of DIAG_NT threads walk tiles of 2^ltx x (256 / 2^ltx) columns, some planes
// at a time. The FP64 pipe is the bound of these marches and takes a warp's
// instruction whole however few of its lanes have a site: the tile is 32 wide unless a
// narrower one, whose warps take two, four or eight rows, has at least 5 % fewer
// warps with a site (sides just above a multiple of 32, or below 32; with fewer
// warps to save the chunks' split of the planes decides: 150 x 101 x 77 is 9 % slower
// 8 wide, with 2 % fewer). us at 32 wide / at the choice, reduction of FP64 fields and
// free energy of FP32 ones: 8 x 512 x 512 2117 / 549, 1299 / 346; 33 x 256 x 256 1147 /
// 645, 681 / 393; 100 x 128 x 128 609 / 493, 348 / 299; 128^3 608, 348 at any width.
constexpr int DIAG_NT = 256, DIAG_LMIN = 2;
constexpr int DIAG_P = ((1 << DIAG_LMIN) + 2) * ((DIAG_NT >> DIAG_LMIN) + 2);  // ring positions of the narrowest tile, the most

inline int diag_tile(int nx, int ny) {
    auto warps = [&](int l) { return (long long)((nx + (1 << l) - 1) >> l) * ((ny + (32 >> l) - 1) / (32 >> l)); };
    int best = 5;
    for (int l = 4; l >= DIAG_LMIN; --l)
        if (20 * warps(l) <= 19 * warps(best)) best = l;
    return best;
}
inline long long diag_tiles(int nx, int ny, int ltx) {
    const int ty = DIAG_NT >> ltx;
    return (long long)((nx + (1 << ltx) - 1) >> ltx) * ((ny + ty - 1) / ty);
}

// planes per tile chunk for nblocks blocks: the even split of nz with the least
// rounds x (planes + extra, for the ring planes' loads and what follows a chunk)
inline int diag_chunk(long long tiles, int nz, int nblocks, double extra) {
    int best = 1;
    double cost = 1e300;
    for (int m = 1; m <= nz; ++m) {
        const int c = (nz + m - 1) / m;
        const double t = (double)((tiles * ((nz + c - 1) / c) + nblocks - 1) / nblocks) * (c + extra);
        if (t < cost) {
            cost = t;
            best = c;
        }
    }
    return best;
}
inline void diag_march(DiagConsts& k, int nblocks) {
    k.ltx = diag_tile(k.nx, k.ny);
    k.chunk = diag_chunk(diag_tiles(k.nx, k.ny, k.ltx), k.nz, nblocks, 1.0);
}

// the constants for handle h (reduce.cu)
void diag_consts(const dl_handle* h, double phi_off, double p_off, DiagConsts& k);

__device__ __forceinline__ int diag_wrap(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

// four planes of u, tile and one-cell ring, component by component
template <typename T>
struct DiagRing {
    T u[4][3][DIAG_P];
};

// What a thread keeps while it marches its column of a tile: plain sums, counts
// as integers, and the moments of w along z, which become those along x and y
// with the column's own x and y once per chunk. Per site that leaves some 25
// FP64 instructions (the sums of w x_a x_b alone took 19 when formed per site),
// fused where a product is added. u comes through shared memory a plane ahead
// (42 of a site's 47 loads are neighbours').
template <typename T>
struct DiagAcc {
    double v, dp, u[3], ke, diss, in, out;  // sums of phi - off, p - off, u, u^2, nu S:S, p - off inside / outside
    double W, Wz, Wzz;
    long long n;
    int vol, nin, nout, bad;
    T vmin, vmax;
};

// |v| is finite, by the bits (a comparison would take the FP64 pipe)
__device__ __forceinline__ bool diag_finite(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ float diag_min(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float diag_max(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double diag_min(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ double diag_max(double a, double b) { return fmax(a, b); }

// site s of plane z, at ring position p (rows ex apart) of planes m, c, n (z - 1, z, z + 1)
template <typename T>
__device__ __forceinline__ void diag_site(const T (&m)[3][DIAG_P], const T (&c)[3][DIAG_P], const T (&n)[3][DIAG_P],
                                          int p, int ex, T v, T dpT, const DiagConsts& k, int z, DiagAcc<T>& a) {
    const double u1 = (double)c[0][p], u2 = (double)c[1][p], u3 = (double)c[2][p];
    const double dp = (double)dpT;
    const double ph = k.phi_off + (double)v;
    // du_b/dx_a: g[b + 3 a]
    T g[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) g[j] = T(0);
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        const T(&r)[3][DIAG_P] = cz(i) < 0 ? m : (cz(i) > 0 ? n : c);
        const int q = p + cy(i) * ex + cx(i);
        const T w[3] = {r[0][q], r[1][q], r[2][q]};
        const int cc[3] = {cx(i), cy(i), cz(i)};
#pragma unroll
        for (int al = 0; al < 3; ++al)
#pragma unroll
            for (int be = 0; be < 3; ++be) {
                if (cc[al] > 0) g[be + 3 * al] += w[be];
                else if (cc[al] < 0) g[be + 3 * al] -= w[be];
            }
    }
    // S:S before the scale, in the storage type (for FP64 fields the FP64 expression)
    const T d01 = g[1] + g[3], d02 = g[2] + g[6], d12 = g[5] + g[7];
    const T sT = T(4) * (g[0] * g[0] + g[4] * g[4] + g[8] * g[8]) + T(2) * (d01 * d01 + d02 * d02 + d12 * d12);
    const double w = (ph - k.phi1) * k.inv_span;
    const double nu = __fma_rn(w, k.dnu, k.nu1);
    a.n += 1;
    a.v += (double)v;
    a.dp += dp;
    a.u[0] += u1;
    a.u[1] += u2;
    a.u[2] += u3;
    a.ke = __fma_rn(u1, u1, a.ke);
    a.ke = __fma_rn(u2, u2, a.ke);
    a.ke = __fma_rn(u3, u3, a.ke);
    a.diss = __fma_rn(nu, (double)sT, a.diss);
    if (ph > k.mid) a.vol += 1;
    if (w > 0.95) {
        a.in += dp;
        a.nin += 1;
    }
    if (w < 0.05) {
        a.out += dp;
        a.nout += 1;
    }
    const double Z = (double)z;
    a.W += w;
    a.Wz = __fma_rn(w, Z, a.Wz);
    a.Wzz = __fma_rn(w, Z * Z, a.Wzz);
    if (!diag_finite(ph)) a.bad += 1;
    a.vmin = diag_min(a.vmin, v);  // NaN is left out
    a.vmax = diag_max(a.vmax, v);
}

// the share of block b of nblocks: its tile chunks in turn; adds the thread's
// sums to acc, folds phi into [vmin, vmax]. All DIAG_NT threads of the block call it.
template <typename T>
__device__ __forceinline__ void diag_sites(const T* __restrict__ mac, const DiagConsts& k, DiagRing<T>& ring, int b,
                                           int nblocks, double (&acc)[DIAG_NSUM], double& vmin, double& vmax) {
    const long long N = k.N, nxy = (long long)k.nx * k.ny;
    const int TX = 1 << k.ltx, TY = DIAG_NT >> k.ltx, EX = TX + 2, np = EX * (TY + 2);
    const int gx = (k.nx + TX - 1) / TX, gy = (k.ny + TY - 1) / TY;
    const long long items = (long long)gx * gy * ((k.nz + k.chunk - 1) / k.chunk);
    const int tid = threadIdx.x, tx = tid & (TX - 1), ty = tid >> k.ltx, p = (ty + 1) * EX + tx + 1;
    DiagAcc<T> a;
    a.v = a.dp = a.u[0] = a.u[1] = a.u[2] = a.ke = a.diss = a.in = a.out = 0.0;
    a.n = 0;
    a.vol = a.nin = a.nout = a.bad = 0;
    a.vmin = T(INFINITY);
    a.vmax = T(-INFINITY);
    for (long long it = b; it < items; it += nblocks) {
        const int bz = (int)(it / (gx * gy)), r = (int)(it - (long long)bz * gx * gy), by = r / gx, bx = r - by * gx;
        const int x = bx * TX + tx, y = by * TY + ty;
        const int z0 = bz * k.chunk, z1 = min(z0 + k.chunk, k.nz);
        const bool act = x < k.nx && y < k.ny;
        const long long col = act ? x + (long long)k.nx * y : 0;
        long long off[2];  // this thread's ring positions tid, tid + DIAG_NT
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int q = tid + j * DIAG_NT, ey = q / EX, ex = q - ey * EX;
            off[j] = (bx * TX - 1 + ex + k.nx) % k.nx + (long long)k.nx * ((by * TY - 1 + ey + k.ny) % k.ny);
        }
        T nu[2][3], nv = T(0), ndp = T(0);  // the plane in flight
        auto fetch = [&](int z) {
            const T* pl = mac + N + nxy * diag_wrap(z, k.nz);
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (tid + j * DIAG_NT < np) nu[j][c] = __ldg(pl + c * N + off[j]);
        };
        auto store = [&](int z) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (tid + j * DIAG_NT < np) ring.u[z & 3][c][tid + j * DIAG_NT] = nu[j][c];
        };
        __syncthreads();  // the previous chunk's readers
        fetch(z0 - 1);
        store(z0 - 1);
        fetch(z0);
        store(z0);
        fetch(z0 + 1);
        nv = __ldg(mac + nxy * z0 + col);
        ndp = __ldg(mac + 4 * N + nxy * z0 + col);
        a.W = a.Wz = a.Wzz = 0.0;
        for (int z = z0; z < z1; ++z) {
            store(z + 1);
            const T v = nv, dp = ndp;
            __syncthreads();
            if (z + 1 < z1) {
                fetch(z + 2);
                nv = __ldg(mac + nxy * (z + 1) + col);
                ndp = __ldg(mac + 4 * N + nxy * (z + 1) + col);
            }
            if (act) diag_site(ring.u[(z - 1) & 3], ring.u[z & 3], ring.u[(z + 1) & 3], p, EX, v, dp, k, z, a);
        }
        const double X = (double)x, Y = (double)y, WX = X * a.W, WY = Y * a.W;
        acc[8] += a.W;
        acc[14] += WX;
        acc[15] += WY;
        acc[16] += a.Wz;
        acc[17] = __fma_rn(X, WX, acc[17]);
        acc[18] = __fma_rn(Y, WY, acc[18]);
        acc[19] += a.Wzz;
        acc[20] = __fma_rn(Y, WX, acc[20]);
        acc[21] = __fma_rn(X, a.Wz, acc[21]);
        acc[22] = __fma_rn(Y, a.Wz, acc[22]);
    }
    acc[13] = acc[8];
    const double n = (double)a.n;
    acc[0] = a.n ? __fma_rn(n, k.phi_off, a.v) : 0.0;
    acc[1] = a.n ? __fma_rn(n, k.p_off, a.dp) : 0.0;
    acc[2] = a.u[0];
    acc[3] = a.u[1];
    acc[4] = a.u[2];
    acc[5] = 0.5 * a.ke;
    acc[6] = 2.0 * k.sfac * a.diss;
    acc[7] = (double)a.vol;
    acc[9] = a.nin ? __fma_rn((double)a.nin, k.p_off, a.in) : 0.0;
    acc[10] = (double)a.nin;
    acc[11] = a.nout ? __fma_rn((double)a.nout, k.p_off, a.out) : 0.0;
    acc[12] = (double)a.nout;
    acc[23] = (double)a.bad;
    // phi_off + v is monotone in v
    if (a.vmin <= a.vmax) {
        vmin = k.phi_off + (double)a.vmin;
        vmax = k.phi_off + (double)a.vmax;
    }
}

}  // namespace dl
