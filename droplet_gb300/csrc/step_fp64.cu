// step_fp64.cu -- the plain form: FP64 storage and arithmetic, evaluated in
// the reference's order so that results are bitwise those of the FP64
// restatement (compiled here with --fmad=false; quotients and sqrt are IEEE
// rounded, by the CUDA operators or by the equal short ways of div_by.cuh).
//
// One time step = two launches:
//   collide_fp64  per site: the record (p0, lap(phi), grad(phi), G, the feq
//                 prefactor A, tau_g, and grad(u) when the LES or Anu terms
//                 need it; program/lbm_drop_xy.f90:590-666 and :576-587,
//                 program/LES_drop_xy.f90:481-502,663-690) in registers, then
//                 feq_i, geq_i (equilibrium_cal :421-476), the collision and
//                 the force (fg_cal :478-515) of the site's own f_i, g_i, each
//                 stored at its destination x + c_i.
//   moments_fp64  per site: the moving-wall bounce-back (drop8_mpi.f90:642-674)
//                 at the wall planes, the moments (physics :541-552) and phi
//                 min/max (:559-574) with one atomic per block; the last block
//                 turns the reduction into the next step's tau_g range.
//
// On GB300 this form is bound by the FP64 pipe, not by HBM (760 bytes per
// site): a warp's FP64 instruction takes the SM 16 cycles, while everything
// else issues in its shadow. What counts is the number of FP64 instructions,
// and the layout follows from it: collided at its own site, a population
// shares c.u, the quadratic terms and the G contraction with its opposite
// (negations and reversed signs are exact) and usq, p0 ... with all 15, where
// a pull from x - c_i evaluates them per direction; the quotients by tau_f,
// tau_g, 3 and the stencil divisors take div_by's one to four instructions
// instead of nine; tau_g is one value on the host where nothing varies it.
// Measured against a record kernel and a collision that pulls from x - c_i
// (ncu, both launches of a step): 64^3 sheared droplet 540 -> 263 us, 128^3
// LES with a force 5.0 -> 2.83 ms; 633 FP64 instructions per site in
// collide_fp64 there and 85 in moments_fp64, the FP64 pipe 85 % busy in both.
#include "dl_internal.cuh"
#include "dl_device.cuh"
#include "div_by.cuh"

#include <string.h>
#include <math.h>

namespace dl {

struct Fp64Args {
    int nx, ny, nz;
    long long N;
    const double* f;   // [15][N]
    const double* g;
    double* fo;
    double* go;
    const double* mac;  // [5][N] phi,u1,u2,u3,p
    double* maco;
    const double* force;  // [3][N]
    DevState* st;
    double kf, kf6, kg, T, a, b;
    double phi1, phi2, nu1, dnu, csd, anu23, anuds;
    DivBy tauf, taug, lapdiv, graddiv, ds;  // taug: the uniform one
    double F0;
    double E[Q], F[Q], Ekf[Q], Ekg[Q], ds3E[Q];
    double wall_bot[5], wall_top[5];  // 6 E_src (U . c_src) terms
    int walls;
    int visc_fixed;
    int les;
    long long step;
};

// classification by the bits: a comparison would take the FP64 pipe
__device__ __forceinline__ bool finite_bits(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool nan_bits(double v) {
    return ((unsigned long long)__double_as_longlong(v) << 1) > 0xFFE0000000000000ull;
}

template <int AL>
__device__ __forceinline__ constexpr int cc(int i) {
    return AL == 0 ? cx(i) : (AL == 1 ? cy(i) : cz(i));
}

// sum_{i=1..14} c_{AL,i} v[i] in the reference's order (the leading 0 and the
// terms with c = 0 add a signed zero, which changes no value)
template <int AL>
__device__ __forceinline__ double csum(const double* v) {
    double s = 0.0;
    bool any = false;
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        if (cc<AL>(i) == 1) s = any ? s + v[i] : v[i];
        else if (cc<AL>(i) == -1) s = s - v[i];
        if (cc<AL>(i) != 0) any = true;
    }
    return s;
}

// (cr1*u1 + cr2*u2) + cr3*u3 with zero terms dropped
__device__ __forceinline__ double cdot(int i, double u1, double u2, double u3) {
    double s = 0.0;
    bool any = false;
    if (cx(i) != 0) { s = cx(i) > 0 ? u1 : -u1; any = true; }
    if (cy(i) != 0) { double t = cy(i) > 0 ? u2 : -u2; s = any ? s + t : t; any = true; }
    if (cz(i) != 0) { double t = cz(i) > 0 ? u3 : -u3; s = any ? s + t : t; any = true; }
    return s;
}

// gtemp = sum_{be} sum_{al} G(al,be) c_al c_be, G(al,be) at G[al + 3 be]
__device__ __forceinline__ double gcontract(int i, const double* G) {
    if (i == 0) return 0.0;
    if (i <= 6) {
        const int al = cx(i) != 0 ? 0 : (cy(i) != 0 ? 1 : 2);
        return G[al + 3 * al];
    }
    const int c[3] = {cx(i), cy(i), cz(i)};
    double s = G[0];
#pragma unroll
    for (int be = 0; be < 3; ++be)
#pragma unroll
        for (int al = 0; al < 3; ++al) {
            if (al + 3 * be == 0) continue;
            s = (c[al] * c[be] > 0) ? s + G[al + 3 * be] : s - G[al + 3 * be];
        }
    return s;
}

// ftemp = sum_{be} sum_{al} (gu(be,al) + gu(al,be)) c_al c_be, gu(a,al) at gu[a + 3 al]
__device__ __forceinline__ double ucontract(int i, const double* gu) {
    const int c[3] = {cx(i), cy(i), cz(i)};
    double s = 0.0;
#pragma unroll
    for (int be = 0; be < 3; ++be)
#pragma unroll
        for (int al = 0; al < 3; ++al) {
            if (c[al] * c[be] == 0) continue;
            const double v = gu[be + 3 * al] + gu[al + 3 * be];
            s = (c[al] * c[be] > 0) ? s + v : s - v;
        }
    return s;
}

__device__ __forceinline__ void site_xyz(long long s, int nx, int ny, int& x, int& y, int& z) {
    const long long t = s / nx;
    x = (int)(s - t * nx);
    z = (int)(t / ny);
    y = (int)(t - (long long)z * ny);
}

// offsets of the planes, rows and columns around a site (wrapped)
struct Around {
    long long xo[3], yo[3], zo[3];
    __device__ __forceinline__ Around(const Fp64Args& a, int x, int y, int z) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            xo[d] = wrapi(x - 1 + d, a.nx);
            yo[d] = (long long)a.nx * wrapi(y - 1 + d, a.ny);
            zo[d] = (long long)a.nx * a.ny * wrapi(z - 1 + d, a.nz);
        }
    }
    // index of x + c_i
    __device__ __forceinline__ long long at(int i) const { return xo[1 + cx(i)] + yo[1 + cy(i)] + zo[1 + cz(i)]; }
};

// the site's record. GU: grad(u) is needed (LES, Anu). SP: the single-phase
// step (no interface terms, tau_g uniform)
template <bool GU, bool SP>
struct Rec64 {
    double ph, U1, U2, U3, P, A, G[9], gu[9];
    double taug, taug_zh, taug_zl;
    int taug_how;
    __device__ __forceinline__ Rec64(const Fp64Args& a, const Around& w, long long s) {
        const long long N = a.N;
        const double* phi = a.mac;
        ph = __ldg(phi + s);
        U1 = __ldg(a.mac + N + s);
        U2 = __ldg(a.mac + 2 * N + s);
        U3 = __ldg(a.mac + 3 * N + s);
        P = __ldg(a.mac + 4 * N + s);
        taug = a.taug.y;
        taug_zh = a.taug.zh;
        taug_zl = a.taug.zl;
        taug_how = a.taug.how;
        A = 0.0;
        if (!SP) {
            double v[Q];
#pragma unroll
            for (int i = 1; i < Q; ++i) v[i] = __ldg(phi + w.at(i));
            const double fun = ph;
            // various_cal :606-613
            const double p0 = fun * a.T / (1.0 - a.b * fun) - a.a * (fun * fun);
            double lap = -(14.0 * fun);
#pragma unroll
            for (int i = 1; i < Q; ++i) lap = lap + v[i];
            lap = div_by(lap, a.lapdiv);
            double gr[3];
            gr[0] = div_by(csum<0>(v), a.graddiv);
            gr[1] = div_by(csum<1>(v), a.graddiv);
            gr[2] = div_by(csum<2>(v), a.graddiv);
            // gphi_cal :655-661
            const double gsq = (gr[0] * gr[0] + gr[1] * gr[1]) + gr[2] * gr[2];
#pragma unroll
            for (int be = 0; be < 3; ++be)
#pragma unroll
                for (int al = 0; al < 3; ++al) {
                    double t = (4.5 * gr[al]) * gr[be];
                    if (al == be) t = t - 1.5 * gsq;
                    G[al + 3 * be] = t;
                }
            // the bracket multiplying F(i) in feq (:453-456)
            A = (p0 - (a.kf * fun) * lap) - a.kf6 * gsq;
        }
        // grad(u) (:623-633)
        if (GU) {
#pragma unroll
            for (int comp = 0; comp < 3; ++comp) {
                const double* uc = a.mac + (1 + comp) * N;
                double q[Q];
#pragma unroll
                for (int i = 1; i < Q; ++i) q[i] = __ldg(uc + w.at(i));
                gu[comp + 0] = div_by(csum<0>(q), a.graddiv);
                gu[comp + 3] = div_by(csum<1>(q), a.graddiv);
                gu[comp + 6] = div_by(csum<2>(q), a.graddiv);
            }
        }
        // tau_g (:576-587; LES :663-690)
        double mn = a.phi1, mx = a.phi2;
        if (!a.visc_fixed) {
            mn = a.st->phi_min;
            mx = a.st->phi_max;
        }
        // with dnu = 0, (phi - mn)/(mx - mn) dnu is 0 (NaN where phi or the range is degenerate)
        const bool flat = a.dnu == 0.0 && mn != mx && finite_bits(ph) && finite_bits(mn) && finite_bits(mx);
        const bool les = GU && a.les;
        if (SP || (flat && !les)) return;
        const double nu = flat ? a.nu1 : (ph - mn) / (mx - mn) * a.dnu + a.nu1;
        double nue = 0.0;
        if (les) {
            double acc = 0.0;
#pragma unroll
            for (int be = 0; be < 3; ++be)
#pragma unroll
                for (int al = 0; al < 3; ++al) {
                    // 0.5 (g + g) = g on the diagonal
                    const double st = al == be ? gu[4 * al] : 0.5 * (gu[al + 3 * be] + gu[be + 3 * al]);
                    acc = al + be ? acc + st * st : st * st;
                }
            nue = a.csd * sqrt(2.0 * acc);
        }
        taug = (0.5 + div_by(3.0 * (nu + nue), a.ds)) + a.anu23;
        taug_how = DIV_GENERAL;
        if (div_divisor_ok(taug)) {
            taug_how = DIV_CORRECT;
            taug_zh = 1.0 / taug;
            taug_zl = div_fma(-taug, taug_zh, 1.0) * taug_zh;
        }
    }
};

// what feq_i and geq_i share: c.u and the G contraction of the representatives
// 0, 1, 2, 3, 7, 8, 9, 10 (an opposite has -c.u and the same contraction)
struct Dirs64 {
    double cu[8], gt[8];
};

// representatives and their opposites
__host__ __device__ constexpr int rep_of(int k) { return k < 4 ? k : k + 3; }  // 0, 1, 2, 3, 7, 8, 9, 10
__host__ __device__ constexpr int opp_of(int i) { return i == 0 ? 0 : (i <= 3 ? i + 3 : i + 4); }

template <bool GU, bool SP>
__device__ __forceinline__ void directions64(const Rec64<GU, SP>& r, Dirs64& d) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int i = rep_of(k);
        d.cu[k] = i == 0 ? 0.0 : cdot(i, r.U1, r.U2, r.U3);
        d.gt[k] = SP ? 0.0 : gcontract(i, r.G);
    }
}

// feq of representative k and of its opposite (equilibrium_cal, program/lbm_drop_xy.f90:452-458)
template <bool GU, bool SP>
__device__ __forceinline__ void feq_pair(const Fp64Args& a, const Rec64<GU, SP>& r, const Dirs64& d, int k,
                                         double (&fe)[2]) {
    const int i = rep_of(k);
    if (i == 0) {
        fe[0] = r.ph + a.F0 * r.A;
        return;
    }
    const double even = a.F[i] * r.A, odd = ((a.E[i] * r.ph) * 3.0) * d.cu[k], gf = a.Ekf[i] * d.gt[k];
    fe[0] = (even + odd) + gf;
    fe[1] = (even - odd) + gf;
}

// geq likewise (:459-469)
template <bool ANU, bool GU, bool SP>
__device__ __forceinline__ void geq_pair(const Fp64Args& a, const Rec64<GU, SP>& r, const Dirs64& d, int k,
                                         double (&ge)[2]) {
    const int i = rep_of(k);
    const double usq = (r.U1 * r.U1 + r.U2 * r.U2) + r.U3 * r.U3;
    const double p3 = 3.0 * r.P, u15 = 1.5 * usq;
    if (i == 0) {
        ge[0] = a.E[0] * (p3 - u15);
        return;
    }
    const double cu = d.cu[k], cu3 = 3.0 * cu, cc45 = 4.5 * (cu * cu);
    double in[2] = {((p3 + cu3) + cc45) - u15, ((p3 - cu3) + cc45) - u15};
    if (ANU) {
        const double t = a.anuds * ucontract(i, r.gu);
        in[0] = in[0] + t;
        in[1] = in[1] + t;
    }
    const double gg = SP ? 0.0 : a.Ekg[i] * d.gt[k];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        ge[q] = a.E[i] * in[q];
        if (!SP) ge[q] = ge[q] + gg;
    }
}

// run body(division) with the division of d's kind: one uniform branch around
// all the quotients by d instead of one at each, where the FP64 instructions
// of the ways not taken would be issued with their predicate off
template <typename B>
__device__ __forceinline__ void with_divisor(const DivBy& d, B&& body) {
    if (d.how == DIV_CORRECT) {
        body([&](double x) { return div_numerator_ok(x) ? div_correct(x, d.y, d.zh, d.zl) : div_general(x, d.y); });
    } else if (d.how == DIV_MARKSTEIN) {
        body([&](double x) { return div_numerator_ok(x) ? div_markstein(x, d.y, d.zh) : div_general(x, d.y); });
    } else if (d.how == DIV_ONE) {
        body([](double x) { return x; });
    } else {
        body([&](double x) { return div_by(x, d); });
    }
}

// ---------------------------------------------------------------------------
// initial populations f <- feq, g <- geq at the site itself (ini :248-251)
template <bool ANU, bool SP>
__global__ void __launch_bounds__(128) equilibrium_fp64(const Fp64Args a) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= a.N) return;
    int x, y, z;
    site_xyz(s, a.nx, a.ny, x, y, z);
    const Rec64<ANU, SP> r(a, Around(a, x, y, z), s);
    Dirs64 d;
    directions64(r, d);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        double e[2];
        if (!SP) {
            feq_pair(a, r, d, k, e);
            a.fo[rep_of(k) * a.N + s] = e[0];
            if (k) a.fo[opp_of(rep_of(k)) * a.N + s] = e[1];
        }
        geq_pair<ANU>(a, r, d, k, e);
        a.go[rep_of(k) * a.N + s] = e[0];
        if (k) a.go[opp_of(rep_of(k)) * a.N + s] = e[1];
    }
}

// ---------------------------------------------------------------------------
template <bool FORCE, bool ANU, bool GU, bool SP>
__global__ void __launch_bounds__(128) collide_fp64(const Fp64Args a) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= a.N) return;
    const long long N = a.N;
    int x, y, z;
    site_xyz(s, a.nx, a.ny, x, y, z);
    const Around w(a, x, y, z);
    const Rec64<GU, SP> r(a, w, s);
    Dirs64 dir;
    directions64(r, dir);
    if (!SP) {
        with_divisor(a.tauf, [&](auto&& over_tauf) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                double fe[2];
                feq_pair(a, r, dir, k, fe);
#pragma unroll
                for (int q = 0; q < (k == 0 ? 1 : 2); ++q) {
                    const int i = q == 0 ? rep_of(k) : opp_of(rep_of(k));
                    const double fs = __ldg(a.f + i * N + s);
                    a.fo[i * N + w.at(i)] = fs - over_tauf(fs - fe[q]);
                }
            }
        });
    }
    double F1 = 0.0, F2 = 0.0, F3 = 0.0;
    if (FORCE) {
        F1 = __ldg(a.force + s);
        F2 = __ldg(a.force + N + s);
        F3 = __ldg(a.force + 2 * N + s);
    }
    const DivBy taug = {r.taug, r.taug_zh, r.taug_zl, r.taug_how};
    with_divisor(taug, [&](auto&& over_taug) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            double ge[2];
            geq_pair<ANU>(a, r, dir, k, ge);
            const double dF = (FORCE && k) ? a.ds3E[rep_of(k)] * cdot(rep_of(k), F1, F2, F3) : 0.0;
#pragma unroll
            for (int q = 0; q < (k == 0 ? 1 : 2); ++q) {
                const int i = q == 0 ? rep_of(k) : opp_of(rep_of(k));
                const double gs = __ldg(a.g + i * N + s);
                double gv = gs - over_taug(gs - ge[q]);
                if (FORCE && k) gv = q == 0 ? gv + dF : gv - dF;
                a.go[i * N + w.at(i)] = gv;
            }
        }
    });
}

// ---------------------------------------------------------------------------
// the streamed populations of a site: bounce-back at the wall planes (stored),
// moments (physics :541-552), phi range. STEP: part of a time step; otherwise
// the moments of given populations alone (a restart)
template <bool STEP, bool SP>
__global__ void __launch_bounds__(256) moments_fp64(const Fp64Args a) {
    const long long s0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const bool active = s0 < a.N;
    const long long s = active ? s0 : 0;
    const long long N = a.N;
    double ph = a.phi1;
    if (!SP) {
        ph = a.fo[s];
#pragma unroll
        for (int i = 1; i < Q; ++i) ph = ph + a.fo[i * N + s];
    }
    double gn[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) gn[i] = a.go[i * N + s];
    if (STEP && a.walls) {
        // bounce_back_LBM, drop8_mpi.f90:651-671 (reference i = 4,8,9,10,15 <- 7,12,13,14,11
        // at the bottom; 7,11,12,13,14 <- 4,15,8,9,10 at the top)
        const long long z = s / ((long long)a.nx * a.ny);
        if (z == 0 || z == a.nz - 1) {
            if (z == 0) {
                gn[3] = gn[6] - a.wall_bot[0];
                gn[7] = gn[11] - a.wall_bot[1];
                gn[8] = gn[12] - a.wall_bot[2];
                gn[9] = gn[13] - a.wall_bot[3];
                gn[14] = gn[10] - a.wall_bot[4];
            }
            if (z == a.nz - 1) {
                gn[6] = gn[3] - a.wall_top[0];
                gn[10] = gn[14] - a.wall_top[1];
                gn[11] = gn[7] - a.wall_top[2];
                gn[12] = gn[8] - a.wall_top[3];
                gn[13] = gn[9] - a.wall_top[4];
            }
            if (active) {
#pragma unroll
                for (int i = 1; i < Q; ++i)
                    if (cz(i) != 0) a.go[i * N + s] = gn[i];
            }
        }
    }
    double pp = div3(gn[0]);
#pragma unroll
    for (int i = 1; i < Q; ++i) pp = pp + div3(gn[i]);
    const double a1 = csum<0>(gn), a2 = csum<1>(gn), a3 = csum<2>(gn);
    bool bad = false;
    if (active) {
        a.maco[s] = ph;
        a.maco[N + s] = a1;
        a.maco[2 * N + s] = a2;
        a.maco[3 * N + s] = a3;
        a.maco[4 * N + s] = pp;
        bad = !(finite_bits(ph) && finite_bits(pp) && finite_bits(a1) && finite_bits(a2) && finite_bits(a3));
    }
    if (!STEP) return;
    // NaN is skipped by the reference's comparisons; exclude it here as well
    const bool in = active && !nan_bits(ph);
    minmax_block_and_finalize<double, true>(a.st, in ? ph : INFINITY, in ? ph : -INFINITY, a.maco, 0.0, N, a.phi1, a.phi2,
                                      bad, a.step, gridDim.x);
}

// ---------------------------------------------------------------------------
static void fill_args(dl_handle* h, Fp64Args& a) {
    const dl_params& P = h->P;
    memset(&a, 0, sizeof(a));
    a.nx = h->nx;
    a.ny = h->ny;
    a.nz = h->nz;
    a.N = (long long)h->N;
    a.st = h->d_state;
    a.kf = P.kappaf;
    a.kf6 = P.kappaf / 6.0;
    a.kg = P.kappag;
    a.T = P.T;
    a.a = P.a;
    a.b = P.b;
    a.phi1 = P.phi1;
    a.phi2 = P.phi2;
    a.nu1 = P.nu1;
    a.dnu = P.nu2 - P.nu1;
    a.csd = P.Cs * P.Cs * P.delta * P.delta;
    a.anu23 = (2.0 / 3.0) * P.Anu;
    a.anuds = P.Anu * P.ds;
    a.tauf = make_div_by(P.tauf);
    a.taug = make_div_by((0.5 + (3.0 * (a.nu1 + 0.0)) / P.ds) + a.anu23);
    a.lapdiv = make_div_by(5.0 * (P.ds * P.ds));
    a.graddiv = make_div_by(10.0 * P.ds);
    a.ds = make_div_by(P.ds);
    a.F0 = h->lc.F[0];
    for (int i = 0; i < Q; ++i) {
        a.E[i] = h->lc.E[i];
        a.F[i] = h->lc.F[i];
        a.Ekf[i] = h->lc.Ekf[i];
        a.Ekg[i] = h->lc.Ekg[i];
        a.ds3E[i] = h->lc.ds3E[i];
    }
    a.walls = P.walls ? 1 : 0;
    a.visc_fixed = (P.visc_mode == DL_VISC_FIXED) ? 1 : 0;
    a.les = P.les ? 1 : 0;
    a.force = h->force64;
}

static inline unsigned nblocks(long long N, int bs) { return (unsigned)((N + bs - 1) / bs); }

int fp64_alloc(dl_handle* h) {
    const size_t N = h->N;
    for (int k = 0; k < 2; ++k) {
        if (!h->single) {  // the single-phase step has no f
            DL_CUDA(h, cudaMalloc(&h->f64[k], sizeof(double) * Q * N));
            DL_CUDA(h, cudaMemsetAsync(h->f64[k], 0, sizeof(double) * Q * N, h->stream));
        }
        DL_CUDA(h, cudaMalloc(&h->g64[k], sizeof(double) * Q * N));
        DL_CUDA(h, cudaMalloc(&h->mac64[k], sizeof(double) * 5 * N));
        DL_CUDA(h, cudaMemsetAsync(h->g64[k], 0, sizeof(double) * Q * N, h->stream));
        DL_CUDA(h, cudaMemsetAsync(h->mac64[k], 0, sizeof(double) * 5 * N, h->stream));
    }
    DL_CUDA(h, cudaMalloc(&h->force64, sizeof(double) * 3 * N));
    DL_CUDA(h, cudaMemsetAsync(h->force64, 0, sizeof(double) * 3 * N, h->stream));
    return DL_OK;
}

void fp64_free(dl_handle* h) {
    for (int k = 0; k < 2; ++k) {
        cudaFree(h->f64[k]);
        cudaFree(h->g64[k]);
        cudaFree(h->mac64[k]);
        h->f64[k] = h->g64[k] = h->mac64[k] = nullptr;
    }
    cudaFree(h->force64);
    h->force64 = nullptr;
}

int fp64_init_equilibrium(dl_handle* h) {
    Fp64Args a;
    fill_args(h, a);
    a.mac = h->mac64[h->cur];
    a.fo = h->f64[h->cur];
    a.go = h->g64[h->cur];
    a.visc_fixed = 1;
    a.les = 0;  // tau_g is not part of an equilibrium
    const unsigned nb = nblocks(a.N, 128);
    if (h->single) DL_LAUNCH(h, false, (equilibrium_fp64<false, true><<<nb, 128, 0, h->stream>>>(a)));
    else if (h->P.Anu != 0.0) DL_LAUNCH(h, false, (equilibrium_fp64<true, false><<<nb, 128, 0, h->stream>>>(a)));
    else DL_LAUNCH(h, false, (equilibrium_fp64<false, false><<<nb, 128, 0, h->stream>>>(a)));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

int fp64_moments_from_populations(dl_handle* h) {
    Fp64Args a;
    fill_args(h, a);
    a.fo = h->f64[h->cur];
    a.go = h->g64[h->cur];
    a.maco = h->mac64[h->cur];
    const unsigned nb = nblocks(a.N, 256);
    if (h->single) DL_LAUNCH(h, false, (moments_fp64<false, true><<<nb, 256, 0, h->stream>>>(a)));
    else DL_LAUNCH(h, false, (moments_fp64<false, false><<<nb, 256, 0, h->stream>>>(a)));
    DL_CUDA(h, cudaGetLastError());
    return DL_OK;
}

template <bool FORCE, bool ANU, bool GU, bool SP>
static void launch_step(dl_handle* h, const Fp64Args& a) {
    DL_LAUNCH(h, true, (collide_fp64<FORCE, ANU, GU, SP><<<nblocks(a.N, 128), 128, 0, h->stream>>>(a)));
    DL_LAUNCH(h, false, (moments_fp64<true, SP><<<nblocks(a.N, 256), 256, 0, h->stream>>>(a)));
}

int fp64_step(dl_handle* h) {
    const int c = h->cur, n = 1 - c;
    const long long step = h->step + 1;
    if (h->force_mode == DL_FORCE_SPECTRAL) {
        int rc = spectral_force_fp64(h, h->mac64[c] + h->N, h->mac64[c] + 2 * h->N, h->mac64[c] + 3 * h->N,
                                     h->force64, h->force64 + h->N, h->force64 + 2 * h->N);
        if (rc != DL_OK) return rc;
    }
    Fp64Args a;
    fill_args(h, a);
    a.f = h->f64[c];
    a.g = h->g64[c];
    a.fo = h->f64[n];
    a.go = h->g64[n];
    a.mac = h->mac64[c];
    a.maco = h->mac64[n];
    a.step = step;
    // wall terms 6 E_src (U . c_src) in the reference's rounding (drop8_mpi.f90:652-670)
    double U[3] = {0.0, 0.0, 0.0};
    if (step >= h->P.wall_start)
        for (int k = 0; k < 3; ++k) U[k] = h->P.wall_u[k];
    const int bot_src[5] = {6, 11, 12, 13, 10}, top_src[5] = {3, 14, 7, 8, 9};
    for (int k = 0; k < 5; ++k) {
        int j = bot_src[k];
        a.wall_bot[k] = 6.0 * h->lc.E[j] * ((-U[0]) * (double)cx(j) + (-U[1]) * (double)cy(j) + (-U[2]) * (double)cz(j));
        j = top_src[k];
        a.wall_top[k] = 6.0 * h->lc.E[j] * ((U[0]) * (double)cx(j) + (U[1]) * (double)cy(j) + (U[2]) * (double)cz(j));
    }
    const bool force = h->force_mode != DL_FORCE_NONE;
    const bool anu = h->P.Anu != 0.0;
    if (h->single) {
        if (force) launch_step<true, false, false, true>(h, a);
        else launch_step<false, false, false, true>(h, a);
    } else if (anu) {
        if (force) launch_step<true, true, true, false>(h, a);
        else launch_step<false, true, true, false>(h, a);
    } else if (a.les) {
        if (force) launch_step<true, false, true, false>(h, a);
        else launch_step<false, false, true, false>(h, a);
    } else {
        if (force) launch_step<true, false, false, false>(h, a);
        else launch_step<false, false, false, false>(h, a);
    }
    DL_CUDA(h, cudaGetLastError());
    h->cur = n;
    h->step = step;
    return DL_OK;
}

}  // namespace dl
