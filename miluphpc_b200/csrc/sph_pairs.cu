// SPH pair sums over the neighbour lists: density, sound speed and pressure,
// the Balsara factors, and the internal (hydro) forces.
//
// The per-neighbour inputs are packed into 32-byte records that one 256-bit
// load fetches (k_pack, once per right-hand side): the loops are gathers, and
// with one 8-byte array per field a pair cost 11 scattered loads.  FP64 pair
// sums read A = (x, y, z, m), B = (v, h), C = (rho, p/rho^2, c_s, m/rho); FP32
// pair sums read A = (FP32 hi of x, h | FP32 lo of x, m) and B = (v, c_s |
// rho, p/rho^2, m/rho, -).  Everything that depends on one particle alone is
// divided out once per particle, not once per pair.
#include "sph.cuh"

namespace {

constexpr int kBlock = 128;

// ------------------------------------------------------------ kernels W
// SmoothingKernel::{spiky, cubicSpline, wendlandc2, wendlandc4, wendlandc6}
// (src/sph/kernel.cu:14-183), 3-D forms, support radius = h.
__device__ __forceinline__ void skernel(int type, double r, double h, double& W, double& dWdr) {
    const double q = r / h;
    W = 0.0;
    dWdr = 0.0;
    switch (type) {
        case 0: {  // spiky
            if (q <= 1.0 && q >= 0.0) {
                const double a = 1.0 - q;
                W = 15. / (M_PI * h * h * h) * a * a * a;
                dWdr = -45 / (M_PI * h * h * h * h) * a * a;
            }
        } break;
        case 1: {  // cubic spline
            const double f = 8. / M_PI * 1. / (h * h * h);
            if (q > 1) {
            } else if (q > 0.5) {
                const double a = 1. - q;
                W = 2. * f * a * a * a;
                dWdr = -6. * f * 1. / h * a * a;
            } else {
                W = f * (6. * q * q * q - 6. * q * q + 1.);
                dWdr = 6. * f / h * (3 * q * q - 2 * q);
            }
        } break;
        case 2: {  // Wendland C2
            if (r <= h) {
                const double a = 1 - q;
                W = 21. / (2 * M_PI * h * h * h) * a * a * a * a * (1 + 4 * q) * (q < 1);
                dWdr = -210. / (M_PI * h * h * h * h) * q * a * a * a * (q < 1);
            }
        } break;
        case 3: {  // Wendland C4 (derivative as written in the reference)
            if (r <= h) {
                const double a = 1 - q, a5 = a * a * a * a * a;
                W = 495. / (32. * M_PI * h * h * h) * a5 * a * (1. + 6. * q + 35. / 3. * q * q) * (q < 1);
                dWdr = -1485. / (16. * M_PI * h * h * h * h) * a5 * (1. - 35. * q * q + 105. * q * q * q) * (q < 1);
            }
        } break;
        default: {  // Wendland C6
            if (r <= h) {
                const double a = 1 - q, a7 = a * a * a * a * a * a * a;
                W = 1365. / (64. * M_PI * h * h * h) * a7 * a * (1. + 8. * q + 25. * q * q + 32 * q * q * q) * (q < 1);
                dWdr = -15015. / (32. * M_PI * h * h * h * h) * q * a7 * (1. + 7 * q + 16 * q * q) * (q < 1);
            }
        } break;
    }
}

// FP32 forms of the same kernels for the mixed-precision pair sums (one
// reciprocal of h, the rest products).
__device__ __forceinline__ void skernel_f(int type, float r, float h, float& W, float& dWdr) {
    const float ih = __frcp_rn(h);
    const float q = r * ih, ih3 = ih * ih * ih, ih4 = ih3 * ih;
    constexpr float kPi = 3.14159265358979f;
    W = 0.f;
    dWdr = 0.f;
    switch (type) {
        case 0: {
            if (q <= 1.f && q >= 0.f) {
                const float a = 1.f - q;
                W = 15.f / kPi * ih3 * a * a * a;
                dWdr = -45.f / kPi * ih4 * a * a;
            }
        } break;
        case 1: {
            const float f = 8.f / kPi * ih3;
            if (q > 1.f) {
            } else if (q > 0.5f) {
                const float a = 1.f - q;
                W = 2.f * f * a * a * a;
                dWdr = -6.f * f * ih * a * a;
            } else {
                W = f * (6.f * q * q * q - 6.f * q * q + 1.f);
                dWdr = 6.f * f * ih * (3.f * q * q - 2.f * q);
            }
        } break;
        case 2: {
            if (q < 1.f) {
                const float a = 1.f - q;
                W = 21.f / (2.f * kPi) * ih3 * a * a * a * a * (1.f + 4.f * q);
                dWdr = -210.f / kPi * ih4 * q * a * a * a;
            }
        } break;
        case 3: {
            if (q < 1.f) {
                const float a = 1.f - q, a5 = a * a * a * a * a;
                W = 495.f / (32.f * kPi) * ih3 * a5 * a * (1.f + 6.f * q + 35.f / 3.f * q * q);
                dWdr = -1485.f / (16.f * kPi) * ih4 * a5 * (1.f - 35.f * q * q + 105.f * q * q * q);
            }
        } break;
        default: {
            if (q < 1.f) {
                const float a = 1.f - q, a7 = a * a * a * a * a * a * a;
                W = 1365.f / (64.f * kPi) * ih3 * a7 * a * (1.f + 8.f * q + 25.f * q * q + 32.f * q * q * q);
                dWdr = -15015.f / (32.f * kPi) * ih4 * q * a7 * (1.f + 7.f * q + 16.f * q * q);
            }
        } break;
    }
}

struct alignas(32) RecD {
    double a, b, c, d;
};
struct alignas(32) RecF {
    float v[8];
};

__device__ __forceinline__ RecD ld_rec(const RecD* p) {
    RecD r;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.a), "=d"(r.b), "=d"(r.c), "=d"(r.d) : "l"(p));
    return r;
}
__device__ __forceinline__ RecF ld_rec(const RecF* p) {
    RecF r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]),
          "=f"(r.v[7])
        : "l"(p));
    return r;
}

// W and dW/dr at one h.  The cubic spline (KERNEL 1) keeps its constants, so
// with one h per particle they are formed once per particle; the other kernels
// (KERNEL -1) are evaluated by type.
template <int KERNEL>
struct KernelD {
    double h, ih, f, g;
    __device__ __forceinline__ void set(double hh) {
        h = hh;
        if (KERNEL == 1) {
            ih = 1.0 / h;
            f = 8. / M_PI / (h * h * h);
            g = 6. * f * ih;
        }
    }
    __device__ __forceinline__ void eval(int type, double r, double& W, double& dWdr) const {
        if (KERNEL == 1) {
            double q = r * ih;
            q = fma(fma(-q, h, r), ih, q);  // r / h rounded once
            const double a = 1. - q;
            const bool outer = q > 0.5;
            W = outer ? 2. * f * a * a * a : f * (6. * q * q * q - 6. * q * q + 1.);
            dWdr = outer ? -g * a * a : g * (3. * q * q - 2. * q);
            if (q > 1.) W = dWdr = 0.0;
        } else {
            skernel(type, r, h, W, dWdr);
        }
    }
};

template <int KERNEL>
struct KernelF {
    float h, ih, f, g;
    __device__ __forceinline__ void set(float hh) {
        h = hh;
        if (KERNEL == 1) {
            ih = __frcp_rn(h);
            f = 8.f / 3.14159265358979f * (ih * ih * ih);
            g = 6.f * f * ih;
        }
    }
    __device__ __forceinline__ void eval(int type, float r, float& W, float& dWdr) const {
        if (KERNEL == 1) {
            const float q = r * ih, a = 1.f - q;
            const bool outer = q > 0.5f;
            W = outer ? 2.f * f * a * a * a : f * (6.f * q * q * q - 6.f * q * q + 1.f);
            dWdr = outer ? -g * a * a : g * (3.f * q * q - 2.f * q);
            if (q > 1.f) W = dWdr = 0.f;
        } else {
            skernel_f(type, r, h, W, dWdr);
        }
    }
};

// r and 1/r from r^2 (r = 0 at r^2 = 0, where 1/r is infinite): one reciprocal
// square root, r corrected by one Newton step
__device__ __forceinline__ void root(double rr, double& r, double& ri) {
    ri = rsqrt(rr);
    r = rr * ri;
    r = fma(fma(-r, r, rr), 0.5 * ri, r);
    if (!(rr > 0.0)) r = 0.0;
}
__device__ __forceinline__ void root(float rr, float& r, float& ri) {
    ri = rsqrtf(rr);
    r = rr * ri;
    r = fmaf(fmaf(-r, r, rr), 0.5f * ri, r);
    if (!(rr > 0.f)) r = 0.f;
}

// T lanes share a particle: lane t (32 / T) + p of a warp takes every T-th list
// entry, from t on, of the warp's particle p
template <int T>
struct Split {
    long s;
    int t;
    __device__ __forceinline__ Split() {
        const int lane = threadIdx.x & 31;
        const long warp = ((long)blockIdx.x * kBlock + threadIdx.x) >> 5;
        s = warp * (32 / T) + (lane & (32 / T - 1));
        t = lane / (32 / T);
    }
    __device__ __forceinline__ double sum(double v) const {
#pragma unroll
        for (int o = 32 / T; o < 32; o <<= 1) v += __shfl_xor_sync(MHPC_FULL, v, o);
        return v;
    }
};

// EOS of one particle (calculateSoundSpeed, then calculatePressure, in the
// reference's order: the ideal-gas sound speed uses the previous pressure)
__device__ __forceinline__ void eos(const MatDev& M, double rho, double e, double& p, double& cs) {
    switch (M.eos_type) {
        case 0: cs = sqrt(M.K * pow(rho, M.gamma - 1.0)); break;
        case 1: case 3: cs = M.cs_init; break;  // constant: initializeSoundSpeed (soundspeed.cu:4-36)
        case 9: cs = sqrt(M.gamma * p / rho); break;
        case 12: cs = 0.0; break;
        default: break;
    }
    switch (M.eos_type) {
        case 0: p = M.K * pow(rho, M.gamma); break;
        case 1: p = (M.bulk / M.n_exp) * (pow(rho / M.rho0, M.n_exp) - 1.0); break;
        case 3: p = 41255.407 * rho; break;
        case 9: p = (M.gamma - 1) * rho * e; break;
        case 12: p = cs * cs * rho; break;
        default: break;
    }
}

// Records A and B from the sorted state (B of the FP32 form is written by the
// density pass, or by k_pack_eos).
__global__ void __launch_bounds__(256) k_pack(SphSorted S, int n, int mixed) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const double x = S.x[s], y = S.y[s], z = S.z[s], m = S.m[s], h = S.h[s];
        if (mixed) {
            const float hx = (float)x, hy = (float)y, hz = (float)z;
            RecF r;
            r.v[0] = hx; r.v[1] = hy; r.v[2] = hz; r.v[3] = (float)h;
            r.v[4] = (float)(x - (double)hx); r.v[5] = (float)(y - (double)hy); r.v[6] = (float)(z - (double)hz);
            r.v[7] = (float)m;
            static_cast<RecF*>(S.ra)[s] = r;
        } else {
            static_cast<RecD*>(S.ra)[s] = RecD{x, y, z, m};
            static_cast<RecD*>(S.rb)[s] = RecD{S.vx[s], S.vy[s], S.vz[s], h};
        }
    }
}

// the records that hold the thermodynamic state of sorted particle s
__device__ __forceinline__ void pack_eos(const SphSorted& S, long s, int mixed, double rho, double p, double cs) {
    if (mixed) {
        RecF r;
        r.v[0] = (float)S.vx[s]; r.v[1] = (float)S.vy[s]; r.v[2] = (float)S.vz[s]; r.v[3] = (float)cs;
        r.v[4] = (float)rho; r.v[5] = (float)(p / (rho * rho)); r.v[6] = (float)(S.m[s] / rho); r.v[7] = 0.f;
        static_cast<RecF*>(S.rb)[s] = r;
    } else {
        static_cast<RecD*>(S.rc)[s] = RecD{rho, p / (rho * rho), cs, S.m[s] / rho};
    }
}

__global__ void __launch_bounds__(256) k_pack_eos(SphSorted S, int n, int mixed) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x)
        pack_eos(S, s, mixed, S.rho[s], S.p[s], S.cs[s]);
}

// --------------------------------------------------- density + EOS (fused)
// calculateDensity (src/sph/density.cu:8-72), then calculateSoundSpeed
// (src/sph/soundspeed.cu:38-97) and calculatePressure (src/sph/pressure.cu:5-87)
// in the reference's order: the ideal-gas sound speed uses the pressure of
// the previous call.  MIXED: FP32 pair terms on neighbour differences formed
// from FP32 hi/lo splits (x_hi = (float)x, x_lo = (float)(x - x_hi), so a
// difference keeps FP32 relative accuracy at any distance from the origin),
// each added to an FP64 sum.
template <bool MIXED, int KERNEL, bool AVG, int T>
__global__ void __launch_bounds__(kBlock) k_density_eos(SphParams P, SphSorted S, const int* __restrict__ nbr,
                                                        const int* __restrict__ noi, const int* __restrict__ perm,
                                                        double* rho_out, double* p_out, double* cs_out,
                                                        DevStatus* st) {
    if (st->code) return;
    const Split<T> L;
    const long s = L.s;
    const bool valid = s < P.n;
    if (T == 1 && !valid) return;
    double rho = 0.0;
    if (P.integrate_density) {
        if (valid) rho = S.rho[s];
    } else {
        if (valid) {
            const int k = min(noi[s], P.maxnb);
            const int* list = nbr + nb_index(s, 0, P.maxnb);
            if (MIXED) {
                const RecF* ra = static_cast<const RecF*>(S.ra);
                const RecF a = ld_rec(ra + s);
                const float hi = a.v[3];
                KernelF<KERNEL> K;
                K.set(hi);
                float W, dWdr;
                if (L.t == 0) {
                    K.eval(P.kernel, 0.f, W, dWdr);
                    rho = (double)(a.v[7] * W);
                }
#pragma unroll 4
                for (int q = L.t; q < k; q += T) {
                    const RecF b = ld_rec(ra + list[(size_t)q * 32]);
                    const float dx = (a.v[0] - b.v[0]) + (a.v[4] - b.v[4]), dy = (a.v[1] - b.v[1]) + (a.v[5] - b.v[5]),
                                dz = (a.v[2] - b.v[2]) + (a.v[6] - b.v[6]);
                    float r, ri;
                    root(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), r, ri);
                    if (AVG) K.set(0.5f * (hi + b.v[3]));
                    K.eval(P.kernel, r, W, dWdr);
                    rho += (double)(b.v[7] * W);
                }
            } else {
                const RecD *ra = static_cast<const RecD*>(S.ra);
                const RecD a = ld_rec(ra + s);
                const double hi = S.h[s];
                KernelD<KERNEL> K;
                K.set(hi);
                double W, dWdr;
                if (L.t == 0) {
                    K.eval(P.kernel, 0.0, W, dWdr);
                    rho = a.d * W;
                }
#pragma unroll 2
                for (int q = L.t; q < k; q += T) {
                    const int j = list[(size_t)q * 32];
                    const RecD b = ld_rec(ra + j);
                    const double dx = a.a - b.a, dy = a.b - b.b, dz = a.c - b.c;
                    double r, ri;
                    root(dx * dx + dy * dy + dz * dz, r, ri);
                    if (AVG) K.set(0.5 * (hi + __ldg(S.h + j)));
                    K.eval(P.kernel, r, W, dWdr);
                    rho += b.d * W;
                }
            }
        }
        rho = L.sum(rho);
        if (valid && !(rho > 0.0)) set_status(st, MHPC_ERR_NAN, (int)s);
    }
    if (!valid || L.t > 0) return;
    const int mid = S.mat ? S.mat[s] : 0;
    double p = S.p[s], cs = S.cs[s];
    eos(P.mat[mid], rho, S.e[s], p, cs);
    S.rho[s] = rho;
    S.p[s] = p;
    S.cs[s] = cs;
    pack_eos(S, s, MIXED, rho, p, cs);
    const int o = perm[s];
    rho_out[o] = rho;
    p_out[o] = p;
    cs_out[o] = cs;
}

// ------------------------------------------------------------- Balsara
// SPH::Kernel::CalcDivvandCurlv (src/sph/kernel.cu:223-342) and the factor of
// internalForces (src/sph/internal_forces.cu:210-217):
//   div v_i = sum_j m_j / rho_j (v_j - v_i) . grad W,
//   curl v_i = sum_j m_j / rho_i (v_i - v_j) x grad W,
//   f_i = |div v_i| / (|div v_i| + |curl v_i| + 1e-4 c_s,i / h_i),
// grad W at h_i (h_bar only under VARIABLE_SML, as in the reference).
__global__ void __launch_bounds__(kBlock) k_balsara(SphParams P, SphSorted S, const int* __restrict__ nbr,
                                                    const int* __restrict__ noi, DevStatus* st) {
    if (st->code) return;
    const long s = (long)blockIdx.x * kBlock + threadIdx.x;
    if (s >= P.n) return;
    const double xi = S.x[s], yi = S.y[s], zi = S.z[s], hi = S.h[s];
    const double vxi = S.vx[s], vyi = S.vy[s], vzi = S.vz[s], rhoi = S.rho[s];
    double divv = 0.0, c0 = 0.0, c1 = 0.0, c2 = 0.0;
    const int k = min(noi[s], P.maxnb);
    for (int q = 0; q < k; ++q) {
        const int j = nbr[nb_index(s, q, P.maxnb)];
        const double hb = P.variable_sml ? 0.5 * (hi + __ldg(S.h + j)) : hi;
        const double dx = xi - __ldg(S.x + j), dy = yi - __ldg(S.y + j), dz = zi - __ldg(S.z + j);
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        double W, dWdr;
        skernel(P.kernel, r, hb, W, dWdr);
        const double g = dWdr / r;
        const double gx = g * dx, gy = g * dy, gz = g * dz;
        const double dvx = vxi - __ldg(S.vx + j), dvy = vyi - __ldg(S.vy + j), dvz = vzi - __ldg(S.vz + j);
        const double mj = __ldg(S.m + j);
        divv += mj / __ldg(S.rho + j) * (-dvx * gx - dvy * gy - dvz * gz);
        const double w = mj / rhoi;
        c0 += w * (dvy * gz - dvz * gy);
        c1 += w * (dvz * gx - dvx * gz);
        c2 += w * (dvx * gy - dvy * gx);
    }
    const double curl = sqrt(c0 * c0 + c1 * c1 + c2 * c2);
    S.bal[s] = fabs(divv) / (fabs(divv) + curl + 1e-4 * S.cs[s] / hi);
}

// ------------------------------------------------------------- forces
// SPH::Kernel::internalForces, hydro part, SPH_EQU_VERSION 1
// (src/sph/internal_forces.cu:372-552).  With g = (dW/dr) / r, d = x_i - x_j,
// dv = v_i - v_j and Pi the viscous pressure of a pair that approaches:
//   s = m_j (p_i/rho_i^2 + p_j/rho_j^2 + Pi),  a_i -= s g d,
//   drho_i/dt = rho_i sum (m_j/rho_j) g d.dv,  de_i/dt = 1/2 sum s g d.dv,
//   dh_i/dt = -(h_i/3) sum (m_j/rho_j) g d.dv.
// With one h per pair (AVG) nothing of the kernel is common to a particle's
// pairs, and W, g and d.dv keep the plain order of operations: in a rigidly
// rotating cloud d.dv is a difference of equal terms, whose value is the
// rounding of that order.
// Bound: the gathers (the records of a warp's lanes lie on lines of their own)
// and, in FP64, the roots and divisions.  Density / forces in us, Sedov lattice,
// with one array per field and every division in the loop, and now: 262,144
// particles FP64 185 / 497 -> 113 / 291; 2,097,152 FP32 773 / 1271 -> 494 / 909.
// The records and the lanes per particle need neighbours to pay for: from 17 on
// density and forces together are faster throughout, with 6 (h = 1.3 spacings) up to a
// fifth slower (2,097,152 FP64: cubic spline 500 -> 431, with h_bar 511 -> 555, Wendland
// C2 498 -> 604).
template <bool MIXED, int KERNEL, bool AVG, int T>
__global__ void __launch_bounds__(kBlock) k_forces(SphParams P, SphSorted S, const int* __restrict__ nbr,
                                                   const int* __restrict__ noi, const int* __restrict__ perm,
                                                   double* ax_o, double* ay_o, double* az_o, double* drhodt_o,
                                                   double* dedt_o, double* dsmldt_o, DevStatus* st) {
    if (st->code) return;
    const Split<T> L;
    const long s = L.s;
    const bool valid = s < P.n;
    if (T == 1 && !valid) return;
    double a0 = 0, a1 = 0, a2 = 0, div = 0, de = 0, rhoi = 0, hid = 0;
    if (valid) {
        const int k = min(noi[s], P.maxnb);
        const int* list = nbr + nb_index(s, 0, P.maxnb);
        const int mid = S.mat ? S.mat[s] : 0;
        if (MIXED) {
            const RecF *ra = static_cast<const RecF*>(S.ra), *rb = static_cast<const RecF*>(S.rb);
            const RecF a = ld_rec(ra + s), v = ld_rec(rb + s);
            const float hi = a.v[3], csi = v.v[3], rhof = v.v[4], pri = v.v[5];
            const float alpha = (float)P.mat[mid].alpha, beta = (float)P.mat[mid].beta;
            const float bali = P.balsara ? (float)S.bal[s] : 1.f;
            KernelF<KERNEL> K;
            K.set(hi);
            rhoi = (double)rhof;
            hid = (double)hi;
#pragma unroll 2
            for (int q = L.t; q < k; q += T) {
                const int j = list[(size_t)q * 32];
                const RecF b = ld_rec(ra + j), w = ld_rec(rb + j);
                const float dx = (a.v[0] - b.v[0]) + (a.v[4] - b.v[4]), dy = (a.v[1] - b.v[1]) + (a.v[5] - b.v[5]),
                            dz = (a.v[2] - b.v[2]) + (a.v[6] - b.v[6]);
                const float rr = dx * dx + dy * dy + dz * dz;
                const float dvx = v.v[0] - w.v[0], dvy = v.v[1] - w.v[1], dvz = v.v[2] - w.v[2];
                const float vr = dvx * dx + dvy * dy + dvz * dz;
                float W, dWdr, g, vw;
                if (AVG) {
                    skernel_f(KERNEL == 1 ? 1 : P.kernel, sqrtf(rr), 0.5f * (hi + b.v[3]), W, dWdr);
                    g = __fdividef(dWdr, sqrtf(rr));
                    vw = dvx * (g * dx) + dvy * (g * dy) + dvz * (g * dz);
                } else {
                    float r, ri;
                    root(rr, r, ri);
                    K.eval(P.kernel, r, W, dWdr);
                    g = dWdr * ri;
                    vw = vr * g;
                }
                float pij = 0.f;
                if (vr < 0.f) {
                    const float csbar = 0.5f * (csi + w.v[3]);
                    const float smooth = 0.5f * (hi + b.v[3]);
                    float mu = __fdividef(smooth * vr, fmaf(smooth * smooth, 1e-2f, rr));
                    if (P.balsara) mu *= 0.5f * (bali + (float)__ldg(S.bal + j));
                    pij = __fdividef((beta * mu - alpha * csbar) * mu, 0.5f * (rhof + w.v[4]));
                }
                const float f = b.v[7] * (pri + w.v[5] + pij), fg = f * g;
                a0 -= (double)(fg * dx);
                a1 -= (double)(fg * dy);
                a2 -= (double)(fg * dz);
                div += (double)(w.v[6] * vw);
                if (P.integrate_energy) de += (double)(f * vw);
            }
        } else {
            const RecD *ra = static_cast<const RecD*>(S.ra), *rb = static_cast<const RecD*>(S.rb),
                       *rc = static_cast<const RecD*>(S.rc);
            const RecD a = ld_rec(ra + s), v = ld_rec(rb + s), c = ld_rec(rc + s);
            const double hi = v.d, csi = c.c, pri = c.b;
            const double alpha = P.mat[mid].alpha, beta = P.mat[mid].beta;
            const double bali = P.balsara ? S.bal[s] : 1.0;
            KernelD<KERNEL> K;
            K.set(hi);
            rhoi = c.a;
            hid = hi;
#pragma unroll 2
            for (int q = L.t; q < k; q += T) {
                const int j = list[(size_t)q * 32];
                const RecD b = ld_rec(ra + j), w = ld_rec(rb + j), cj = ld_rec(rc + j);
                const double dx = a.a - b.a, dy = a.b - b.b, dz = a.c - b.c;
                const double rr = dx * dx + dy * dy + dz * dz;
                const double dvx = v.a - w.a, dvy = v.b - w.b, dvz = v.c - w.c;
                const double vr = dvx * dx + dvy * dy + dvz * dz;
                double W, dWdr, g, vw;
                if (AVG) {
                    skernel(KERNEL == 1 ? 1 : P.kernel, sqrt(rr), 0.5 * (hi + w.d), W, dWdr);
                    g = dWdr / sqrt(rr);
                    vw = dvx * (g * dx) + dvy * (g * dy) + dvz * (g * dz);
                } else {
                    double r, ri;
                    root(rr, r, ri);
                    K.eval(P.kernel, r, W, dWdr);
                    g = dWdr * ri;
                    vw = vr * g;
                }
                double pij = 0.0;
                if (vr < 0) {
                    const double csbar = 0.5 * (csi + cj.c);
                    const double smooth = 0.5 * (hi + w.d);
                    double mu = smooth * vr / (rr + smooth * smooth * 1e-2);
                    if (P.balsara) mu *= (bali + __ldg(S.bal + j)) / 2.;
                    pij = (beta * mu - alpha * csbar) * mu / (0.5 * (rhoi + cj.a));
                }
                const double f = b.d * (pri + cj.b + pij), fg = f * g;
                a0 -= fg * dx;
                a1 -= fg * dy;
                a2 -= fg * dz;
                div += cj.d * vw;
                if (P.integrate_energy) de += f * vw;
            }
        }
    }
    if (T > 1) {
        a0 = L.sum(a0); a1 = L.sum(a1); a2 = L.sum(a2); div = L.sum(div);
        if (P.integrate_energy) de = L.sum(de);
    }
    if (!valid || L.t > 0) return;
    const int o = perm[s];
    ax_o[o] = a0;
    ay_o[o] = a1;
    az_o[o] = a2;
    if (drhodt_o) drhodt_o[o] = rhoi * div;
    if (dedt_o) dedt_o[o] = 0.5 * de;
    if (dsmldt_o) dsmldt_o[o] = P.integrate_sml ? -(1. / 3.) * hid * div : 0.0;
}

// Lanes per particle of the pair loops.  More lanes shorten the chain of
// dependent gathers of a small n; many lose to the sums across lanes.
// Density / forces in us with 1, 2 and 4 lanes: 35,937 particles FP32 41 / 51,
// 29 / 29, 22 / 27; 262,144 FP64 144 / 333, 113 / 291, 109 / 301; 2,097,152 FP32
// 494 / 969, 543 / 909, 607 / 985.
int pair_lanes(int n, bool density_f32) {
    if (n <= 65536) return 4;
    return density_f32 && n > 500000 ? 1 : 2;
}

template <bool MIXED, int KERNEL, bool AVG>
void density_eos(const SphParams& P, const SphSorted& S, const int* nbr, const int* noi, const int* perm,
                 double* rho, double* p, double* cs, DevStatus* st, cudaStream_t s) {
    const int t = pair_lanes(P.n, MIXED);
    const int blocks = (int)(((long)P.n * t + kBlock - 1) / kBlock);
    if (t == 4) k_density_eos<MIXED, KERNEL, AVG, 4><<<blocks, kBlock, 0, s>>>(P, S, nbr, noi, perm, rho, p, cs, st);
    else if (t == 2) k_density_eos<MIXED, KERNEL, AVG, 2><<<blocks, kBlock, 0, s>>>(P, S, nbr, noi, perm, rho, p, cs, st);
    else k_density_eos<MIXED, KERNEL, AVG, 1><<<blocks, kBlock, 0, s>>>(P, S, nbr, noi, perm, rho, p, cs, st);
}

template <bool MIXED, int KERNEL, bool AVG>
void forces(const SphParams& P, const SphSorted& S, const int* nbr, const int* noi, const int* perm, double* ax,
            double* ay, double* az, double* drhodt, double* dedt, double* dsmldt, DevStatus* st, cudaStream_t s) {
    const int t = pair_lanes(P.n, false);
    const int blocks = (int)(((long)P.n * t + kBlock - 1) / kBlock);
    if (t == 4) k_forces<MIXED, KERNEL, AVG, 4><<<blocks, kBlock, 0, s>>>(P, S, nbr, noi, perm, ax, ay, az, drhodt,
                                                                       dedt, dsmldt, st);
    else k_forces<MIXED, KERNEL, AVG, 2><<<blocks, kBlock, 0, s>>>(P, S, nbr, noi, perm, ax, ay, az, drhodt, dedt,
                                                                  dsmldt, st);
}

// the instance of F for the configuration
#define MHPC_PAIR(F, ...)                                                                   \
    do {                                                                                    \
        if (P.kernel == 1) {                                                                \
            if (P.mixed && P.avg_h) F<true, 1, true>(__VA_ARGS__);                          \
            else if (P.mixed) F<true, 1, false>(__VA_ARGS__);                               \
            else if (P.avg_h) F<false, 1, true>(__VA_ARGS__);                               \
            else F<false, 1, false>(__VA_ARGS__);                                           \
        } else {                                                                            \
            if (P.mixed && P.avg_h) F<true, -1, true>(__VA_ARGS__);                         \
            else if (P.mixed) F<true, -1, false>(__VA_ARGS__);                              \
            else if (P.avg_h) F<false, -1, true>(__VA_ARGS__);                              \
            else F<false, -1, false>(__VA_ARGS__);                                          \
        }                                                                                   \
    } while (0)

}  // namespace

int sph_density_eos(const SphParams& P, const SphSorted& S, const int* nbr, const int* noi, const int* perm,
                    double* rho_out, double* p_out, double* cs_out, DevStatus* st, cudaStream_t s) {
    if (P.n <= 0) return MHPC_OK;
    k_pack<<<grid_for(P.n, 256, 148 * 8), 256, 0, s>>>(S, P.n, P.mixed);
    MHPC_PAIR(density_eos, P, S, nbr, noi, perm, rho_out, p_out, cs_out, st, s);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}

int sph_balsara(const SphParams& P, const SphSorted& S, const int* nbr, const int* noi, DevStatus* st,
                cudaStream_t s) {
    if (P.n <= 0) return MHPC_OK;
    k_balsara<<<(P.n + kBlock - 1) / kBlock, kBlock, 0, s>>>(P, S, nbr, noi, st);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}

int sph_forces(const SphParams& P, const SphSorted& S, bool packed, const int* nbr, const int* noi, const int* perm,
               double* ax, double* ay, double* az, double* drhodt, double* dedt, double* dsmldt, DevStatus* st,
               cudaStream_t s) {
    if (P.n <= 0) return MHPC_OK;
    if (!packed) {
        k_pack<<<grid_for(P.n, 256, 148 * 8), 256, 0, s>>>(S, P.n, P.mixed);
        k_pack_eos<<<grid_for(P.n, 256, 148 * 8), 256, 0, s>>>(S, P.n, P.mixed);
    }
    MHPC_PAIR(forces, P, S, nbr, noi, perm, ax, ay, az, drhodt, dedt, dsmldt, st, s);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}
