// rb_solve.cuh -- in-group accelerators and the group loop, run by one team (cluster) per problem.
//
// Restates on the device: livolant! (src/tools/livolant.jl:110-154), anderson!
// (src/tools/anderson.jl:38-140), gmres! (src/tools/gmres.jl:35-133), bicgstab!
// (src/tools/bicgstab.jl:30-101), sn_one_speed (sn_one_speed.jl:81-195) and the group loop of
// compute_flux(::SN) (sn_flux.jl:146-224). Every scalar decision (convergence tests,
// Hessenberg, Givens, Anderson normal equations) is taken from team reductions whose bits are
// identical in every thread, so all threads of the cluster branch together; each CTA keeps its
// own copy of the small scalar arrays, updated by its leader thread.
#pragma once
#include <math_constants.h>

#include "rb_kernels.cuh"
#include "rb_local1d.cuh"
#include "rb_sweep_oct.cuh"

namespace rb {

struct SolveStat {
    int iter;
    double resid;
    int conv;
    double rho;
};

__device__ __forceinline__ double rho_estimate(double r0, double r, int it) {  // krylov_state.jl:139-144
    if (it > 1 && r0 > 0.0 && r > 0.0) return pow(r / r0, 1.0 / (it - 1));
    return CUDART_NAN;
}

// LO: the team runs only 1D problems on the local pass (the kernel that carries no other pass)
template <class Team, bool LO = false>
struct Solver {
    Team &t;
    const DevProblem &P;
    GroupShared &gs;
    int ig;
    const double *phiE_in;
    double *phiE_out;
    long long npass;
    void *local = nullptr;  // shared-memory region of the local 1D pass (and of the 3D octant sweep)
    long long local_bytes = 0;
    int local_ok = 0;       // this problem takes the local 1D pass
    int local_w = 0;        // and keeps the slice of w in shared memory in the Gram-Schmidt loop

    __device__ double *vec(int k) const { return P.vecs + (long long)k * P.vstride; }

    // load_and_pass! (sn_one_speed.jl:138-143): out <- T(zin)
    // The mixed form runs every pass with FP32 angular arithmetic except two per group
    // (final = 1), which are FP64: the Krylov right-hand side c = T(0) and the reconstruction
    // pass, which produces the returned flux moments and the energy-face flux carried into the
    // next group (the outer defect-correction update).
    // One copy of the pass per kernel (it is called from every accelerator): its own register
    // allocation, and a compile time that does not grow with the number of call sites.
    // emit: the outgoing energy-face flux is written (the reconstruction pass alone: the others' is
    // never read).
    __device__ __noinline__ void pass(const double *zin, double *out, int homog, int mv, int final = 0, int emit = 0) {
        const int mixed = (P.precision == 1 && !final) ? 1 : 0;
        double *phiE_out = emit ? this->phiE_out : nullptr;
        npass++;
        if constexpr (std::is_same<Team, ClusterTeam>::value) {
            if (LO || local_ok) {
                pass1d_local(t, P, gs, zin, out, homog, mv, ig, phiE_in, phiE_out, mixed);
                return;
            }
        }
        if constexpr (std::is_same<Team, GridTeam>::value) {  // the grid team runs 2D/3D problems only
            pass_md(t, P, gs, local, local_bytes, zin, out, homog, mv, ig, phiE_in, phiE_out, mixed);
        } else if constexpr (!LO) {
            if (P.ndims == 1) pass1d(t, P, gs, local, local_bytes, zin, out, homog, mv, ig, phiE_in, phiE_out, mixed);
            else pass_md(t, P, gs, local, local_bytes, zin, out, homog, mv, ig, phiE_in, phiE_out, mixed);
        }
    }
    __device__ void fixedpoint(double *out, const double *zin) { pass(zin, out, 0, 0); }
    // matvec! (sn_one_speed.jl:147): out <- zin − A·zin
    __device__ void matvec(double *out, const double *zin) { pass(zin, out, 1, 1); }
    __device__ double norm(const double *a) { return sqrt(vdot(t, a, a, P.nstate)); }

    // ---------------------------------------------------------------- livolant (and "none")
    __device__ __noinline__ SolveStat livolant(double *z, int maxit, double tol, int period) {
        const long long N = P.nstate;
        double *g = vec(1), *z1 = vec(3), *z0 = vec(4);
        int nhist = 0, iter = 0, conv = 0;
        double resid = 1.0, resid0 = CUDART_NAN;
        for (int it = 1; it <= maxit; it++) {
            fixedpoint(g, z); iter++;
            // ‖g − z‖ and ‖g‖ in one reduction
            double v[2] = {0.0, 0.0};
            for (long long i = t.rank(); i < N; i += t.size()) {
                const double f = g[i] + (-1.0) * z[i];
                v[0] += f * f; v[1] += g[i] * g[i];
            }
            t.template sumk<2>(v);
            resid = sqrt(v[0]) / fmax(sqrt(v[1]), 1e-16);
            if (isnan(resid0)) resid0 = resid;
            if (resid < tol) { vcopy(t, z, g, N); conv = 1; break; }
            if (period > 0 && it % period == 0 && nhist >= 2) {
                double w[2] = {0.0, 0.0};
                for (long long i = t.rank(); i < N; i += t.size()) {
                    const double e0 = z1[i] - z0[i], e1 = g[i] - z1[i], de = e1 - e0;
                    w[0] += e0 * de; w[1] += de * de;
                }
                t.template sumk<2>(w);
                double mu = 1.0;
                if (w[1] != 0.0) { mu = -w[0] / w[1]; if (mu <= 0) mu = 1.0; }
                for (long long i = t.rank(); i < N; i += t.size()) {
                    z[i] = g[i] * mu + (1.0 - mu) * z1[i];
                    z0[i] = z1[i];
                    z1[i] = g[i];
                }
            } else {
                for (long long i = t.rank(); i < N; i += t.size()) {
                    z[i] = g[i];
                    z0[i] = z1[i];
                    z1[i] = g[i];
                }
            }
            t.sync();
            nhist++;
        }
        SolveStat s = {iter, resid, conv, rho_estimate(resid0, resid, iter)};
        return s;
    }

    // ---------------------------------------------------------------- anderson (β = 1)
    __device__ __noinline__ SolveStat anderson(double *z, int depth, int maxit, double tol) {
        const long long N = P.nstate;
        const int m = depth > 1 ? depth : 1;
        double *g = vec(1), *f = vec(2), *fo = vec(3), *go = vec(4);
        // history ring: logical i -> slot (head + i) % m; ΔF slot s = vec(5+s), ΔG = vec(5+m+s)
        int nh = 0, head = 0, iter = 0, conv = 0;
        double resid = 1.0, resid0 = CUDART_NAN;
        for (int it = 1; it <= maxit; it++) {
            fixedpoint(g, z); iter++;
            double v[3] = {0.0, 0.0, 0.0};
            for (long long i = t.rank(); i < N; i += t.size()) {
                const double fi = g[i] + (-1.0) * z[i];
                f[i] = fi;
                v[0] += fi * fi; v[1] += z[i] * z[i]; v[2] += g[i] * g[i];
            }
            t.template sumk<3>(v);
            resid = sqrt(v[0]) / fmax(fmax(sqrt(v[1]), sqrt(v[2])), 1e-16);
            if (isnan(resid0)) resid0 = resid;
            if (resid < tol) { conv = 1; break; }
            if (it == 1) {
                vaxpy(t, 1.0, f, z, N);
            } else {
                if (nh == m) { head = (head + 1) % m; nh--; }  // popfirst!
                const int slot = (head + nh) % m;
                double *dF = vec(5 + slot), *dG = vec(5 + m + slot);
                for (long long i = t.rank(); i < N; i += t.size()) {
                    dF[i] = f[i] + (-1.0) * fo[i];
                    dG[i] = g[i] + (-1.0) * go[i];
                }
                t.sync();
                nh++;
                const int mk = nh;
                for (int i = 0; i < mk; i++) {
                    const double *dFi = vec(5 + (head + i) % m);
                    double bi = vdot(t, dFi, f, N);
                    if (t.leader()) gs.b[i] = bi;
                    for (int j = 0; j < mk; j++) {
                        double aij = vdot(t, dFi, vec(5 + (head + j) % m), N);
                        if (t.leader()) gs.A[i + mk * j] = aij;
                    }
                }
                __syncthreads();
                if (t.leader()) {
                    double *A = gs.A, *x = gs.b;
                    double tr = 0.0;
                    for (int i = 0; i < mk; i++) tr += A[i + mk * i];
                    const double lam = 1e-12 * (tr / mk + 1e-300);
                    for (int i = 0; i < mk; i++) A[i + mk * i] += lam;
                    const int n = mk;  // anderson_solve (anderson.jl:112-140)
                    for (int k = 0; k < n; k++) {
                        int p = k; double mx = fabs(A[k + n * k]);
                        for (int i = k + 1; i < n; i++) if (fabs(A[i + n * k]) > mx) { mx = fabs(A[i + n * k]); p = i; }
                        if (p != k) {
                            for (int j = k; j < n; j++) { double tt = A[k + n * j]; A[k + n * j] = A[p + n * j]; A[p + n * j] = tt; }
                            double tt = x[k]; x[k] = x[p]; x[p] = tt;
                        }
                        const double piv = A[k + n * k];
                        if (piv == 0.0) continue;
                        for (int i = k + 1; i < n; i++) {
                            const double fac = A[i + n * k] / piv;
                            for (int j = k; j < n; j++) A[i + n * j] -= fac * A[k + n * j];
                            x[i] -= fac * x[k];
                        }
                    }
                    for (int k = n - 1; k >= 0; k--) {
                        double s = x[k];
                        for (int j = k + 1; j < n; j++) s -= A[k + n * j] * x[j];
                        x[k] = A[k + n * k] != 0.0 ? s / A[k + n * k] : 0.0;
                    }
                }
                __syncthreads();
                // z ← z + f − Σ γ_i ΔG_i  (β = 1: the ΔF term carries a zero factor)
                for (long long i = t.rank(); i < N; i += t.size()) {
                    double zi = z[i] + 1.0 * f[i];
                    for (int k = 0; k < mk; k++) zi += -gs.b[k] * vec(5 + m + (head + k) % m)[i];
                    z[i] = zi;
                }
                t.sync();
            }
            for (long long i = t.rank(); i < N; i += t.size()) { fo[i] = f[i]; go[i] = g[i]; }
            t.sync();
        }
        SolveStat s = {iter, resid, conv, rho_estimate(resid0, resid, iter)};
        return s;
    }

    // Modified Gram-Schmidt of w against V_0..V_jb (gmres.jl) in two reductions instead of jb + 2.
    // The coefficients of the modified form, h_i = V_i·(w − Σ_{k<i} h_k V_k), are the solution of
    // (I + L)·h = Vᵀw with L the strictly lower part of VᵀV (Świrydowicz, Langou, Ananthan, Yang and
    // Thomas 2021, "Low synchronization Gram-Schmidt and GMRES algorithms"): same projection and same
    // stability, every inner product from one pass over the basis, and no basis vector's load waits
    // for a reduction. L's row of V_jb comes with the products of w and stays below the diagonal of
    // H, which the Givens rotations leave free. A step of a 200-cell, S16 slab on 4 CTAs: 41 us step by
    // step, 10 here (the two reductions 4, the rest loads); 128×128, S12: 288 and 140. Writes H[0..jb, jb] and V_{jb+1}; returns
    // H[jb+1, jb].
    //
    // Each thread takes elements q0, q0 + blockDim.x, … < q1 (of type E: a double or an aligned
    // pair); Krylov vectors hold element q at [q], w is read at w0 and written at w1 (shared memory
    // on the local 1D pass).
    static __device__ __forceinline__ double dot_add(double s, double a, double b) { return s + a * b; }
    static __device__ __forceinline__ double dot_add(double s, double2 a, double2 b) { return (s + a.x * b.x) + a.y * b.y; }
    static __device__ __forceinline__ double minus(double a, double h, double v) { return a - h * v; }
    static __device__ __forceinline__ double2 minus(double2 a, double h, double2 v) {
        return make_double2(a.x - h * v.x, a.y - h * v.y);
    }
    static __device__ __forceinline__ double times(double a, double s) { return a * s; }
    static __device__ __forceinline__ double2 times(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

    // acc[e] += V_{i0+e}·w and acc[4+e] += V_{i0+e}·V_jb over this thread's elements: four basis
    // vectors at a time, U elements' loads in flight together
    template <typename E, int U>
    static __device__ __forceinline__ void mgs_dots(const E *w, const E *vj, const E *const (&V)[4], int q0, int q1,
                                                    double (&acc)[8]) {
        const int step = blockDim.x;
        int q = q0;
        for (; q + (U - 1) * step < q1; q += U * step) {
            E xw[U], xj[U], xv[U][4];
#pragma unroll
            for (int u = 0; u < U; u++) {
                xw[u] = w[q + u * step];
                xj[u] = vj[q + u * step];
#pragma unroll
                for (int e = 0; e < 4; e++) xv[u][e] = V[e][q + u * step];
            }
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    acc[e] = dot_add(acc[e], xw[u], xv[u][e]);
                    acc[4 + e] = dot_add(acc[4 + e], xj[u], xv[u][e]);
                }
        }
        for (; q < q1; q += step) {
            E x[6] = {w[q], vj[q], V[0][q], V[1][q], V[2][q], V[3][q]};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                acc[e] = dot_add(acc[e], x[0], x[2 + e]);
                acc[4 + e] = dot_add(acc[4 + e], x[1], x[2 + e]);
            }
        }
    }

    // w1 = w0 − Σ h_i V_i over this thread's elements; returns its part of ‖w1‖²
    template <typename E, int U>
    static __device__ __forceinline__ double mgs_update(const E *w0, E *w1, const E *V0, long long ldv, int q0, int q1, int n,
                                                        const double *h) {
        const int step = blockDim.x;
        double s = 0.0;
        for (int q = q0; q < q1; q += U * step) {
            E x[U];
            int g[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                g[u] = q + u * step < q1 ? q + u * step : q;
                x[u] = w0[g[u]];
            }
            int i = 0;
            for (; i + 4 <= n; i += 4) {
                E v[4][U];
#pragma unroll
                for (int e = 0; e < 4; e++)
#pragma unroll
                    for (int u = 0; u < U; u++) v[e][u] = V0[(i + e) * ldv + g[u]];
#pragma unroll
                for (int e = 0; e < 4; e++)
#pragma unroll
                    for (int u = 0; u < U; u++) x[u] = minus(x[u], h[i + e], v[e][u]);
            }
            if (i < n) {
                E v[3][U];
#pragma unroll
                for (int e = 0; e < 3; e++)
#pragma unroll
                    for (int u = 0; u < U; u++) v[e][u] = V0[min(i + e, n - 1) * ldv + g[u]];
#pragma unroll
                for (int e = 0; e < 3; e++)
                    if (i + e < n)
#pragma unroll
                        for (int u = 0; u < U; u++) x[u] = minus(x[u], h[i + e], v[e][u]);
            }
#pragma unroll
            for (int u = 0; u < U; u++)
                if (q + u * step < q1) {
                    w1[g[u]] = x[u];
                    s = dot_add(s, x[u], x[u]);
                }
        }
        return s;
    }

    template <typename E>
    static __device__ __forceinline__ void mgs_scale(const E *w, E *v, double inv, int q0, int q1) {
        const int step = blockDim.x;
        for (int q = q0; q < q1; q += 4 * step) {
            E x[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (q + u * step < q1) x[u] = w[q + u * step];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (q + u * step < q1) v[q + u * step] = times(x[u], inv);
        }
    }

    // h from b = Vᵀw by forward substitution with I + L (one warp, a row or two per lane)
    __device__ __forceinline__ void mgs_coefficients(double *b, int n, int m) {
        double *H = gs.H;
        const int jb = n - 1, lane = threadIdx.x & 31;
        if (threadIdx.x < 32) {
            for (int i = lane; i < jb; i += 32) H[jb + (m + 1) * i] = b[n + i];
            __syncwarp();
            double b0 = lane < n ? b[lane] : 0.0, b1 = lane + 32 < n ? b[lane + 32] : 0.0;
            for (int k = 0; k < jb; k++) {
                const double hk = __shfl_sync(0xffffffffu, k < 32 ? b0 : b1, k & 31);
                if (lane > k && lane < n) b0 -= H[lane + (m + 1) * k] * hk;
                if (lane + 32 > k && lane + 32 < n) b1 -= H[lane + 32 + (m + 1) * k] * hk;
            }
            if (lane < n) { b[lane] = b0; H[lane + (m + 1) * jb] = b0; }
            if (lane + 32 < n) { b[lane + 32] = b1; H[lane + 32 + (m + 1) * jb] = b1; }
        }
        __syncthreads();
    }

    // The mixed form keeps the modified form step by step (its FP32 roundings follow the last bit of
    // every coefficient): w − h_i V_i fused with the product of the next basis vector. On the local 1D
    // pass w, V_i and V_{i+1} are slices in shared memory (ψ's region is free meanwhile), V_{i+1}
    // copied asynchronously while the reduction of h_i is under way: short rolled loops, no register
    // arrays (40 elements a thread in registers spilled, and the unrolled loops took 40 predicated
    // turns for slices of 3). Where the third slice does not fit, V_{i+1} is loaded in the update.
    __device__ __noinline__ double mgs_ordered(double *w, int jb, int m) {
        const Local1D &L = *reinterpret_cast<const Local1D *>(gs.l1d);
        const long long ldv = P.vstride, e0 = L.e0, eb = L.eb - L.l1;
        const double *V = vec(4);
        const int ls = L.ls, l1 = L.l1, tid = threadIdx.x;
        constexpr int step = RB_THREADS;
        double *ws = L.ws, *va = reinterpret_cast<double *>(L.psi), *vb = L.vb, acc[1] = {0.0};
        auto at = [=](int j) -> long long { return (j < l1 ? e0 : eb) + j; };
        auto copy = [&](double *dst, const double *src) {
#pragma unroll 4
            for (int j = tid; j < ls; j += step) cp_zfill<8>(dst + j, src + at(j), true);
        };
        auto landed = [] {
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        };
        copy(ws, w);
        copy(va, V);
        landed();
#pragma unroll 8
        for (int j = tid; j < ls; j += step) acc[0] += ws[j] * va[j];
        for (int i = 0; i <= jb; i++) {
            const double *Vn = V + (i + 1) * ldv;
            if (vb && i < jb) copy(vb, Vn);
            t.template sumk<1>(acc);
            const double h = acc[0];
            if (t.leader()) gs.H[i + (m + 1) * jb] = h;
            acc[0] = 0.0;
            landed();
            if (i == jb) {
#pragma unroll 8
                for (int j = tid; j < ls; j += step) {
                    const double x = ws[j] + (-h) * va[j];
                    ws[j] = x;
                    acc[0] += x * x;
                }
            } else if (vb) {
#pragma unroll 8
                for (int j = tid; j < ls; j += step) {
                    const double x = ws[j] + (-h) * va[j];
                    ws[j] = x;
                    acc[0] += x * vb[j];
                }
                double *s = va;
                va = vb;
                vb = s;
            } else {
                for (int j0 = tid; j0 < ls; j0 += 8 * step) {
                    double b[8];
#pragma unroll
                    for (int u = 0; u < 8; u++)
                        if (j0 + u * step < ls) b[u] = Vn[at(j0 + u * step)];
#pragma unroll
                    for (int u = 0; u < 8; u++)
                        if (j0 + u * step < ls) {
                            const int j = j0 + u * step;
                            const double x = ws[j] + (-h) * va[j];
                            ws[j] = x;
                            va[j] = b[u];
                            acc[0] += x * b[u];
                        }
                }
            }
        }
        t.template sumk<1>(acc);
        const double hn = sqrt(acc[0]);
        if (hn > 0.0) {
            const double inv = 1.0 / hn;
            double *Vo = vec(4 + jb + 1);
#pragma unroll 4
            for (int j = tid; j < ls; j += step) Vo[at(j)] = ws[j] * inv;
        }
        return hn;
    }
    // the same over 16-byte pairs of the CTA's contiguous range
    __device__ __forceinline__ double mgs_ordered_pairs(double *w, int jb, int m) {
        const long long N2 = P.vstride / 2;
        double h = vdot2(t, w, vec(4), N2);
        double2 *w2 = RB_D2(w);
        for (int i = 0; i <= jb; i++) {
            if (t.leader()) gs.H[i + (m + 1) * jb] = h;
            const double2 *Vi2 = RB_CD2(vec(4 + i)), *Vn2 = i < jb ? RB_CD2(vec(4 + i + 1)) : nullptr;
            double acc[1] = {0.0};
            double2 xw[4], xv[4], xn[4];
            if (Vn2) {
                RB_VPAIRS_D(t, N2, 4, { xw[u_] = w2[q]; xv[u_] = Vi2[q]; xn[u_] = Vn2[q]; }, {
                    double2 wq;
                    wq.x = xw[u_].x + (-h) * xv[u_].x;
                    wq.y = xw[u_].y + (-h) * xv[u_].y;
                    w2[q] = wq;
                    acc[0] += wq.x * xn[u_].x;
                    acc[0] += wq.y * xn[u_].y;
                })
            } else {
                RB_VPAIRS_D(t, N2, 4, { xw[u_] = w2[q]; xv[u_] = Vi2[q]; }, {
                    double2 wq;
                    wq.x = xw[u_].x + (-h) * xv[u_].x;
                    wq.y = xw[u_].y + (-h) * xv[u_].y;
                    w2[q] = wq;
                    acc[0] += wq.x * wq.x;
                    acc[0] += wq.y * wq.y;
                })
            }
            t.template sumk<1>(acc);
            h = acc[0];
        }
        const double hn = sqrt(h);
        if (hn > 0.0) {
            const double inv = 1.0 / hn;
            double2 *Vn2 = RB_D2(vec(4 + jb + 1));
            double2 xw[4];
            RB_VPAIRS_D(t, N2, 4, { xw[u_] = w2[q]; }, { Vn2[q] = make_double2(xw[u_].x * inv, xw[u_].y * inv); })
        }
        return hn;
    }
    __device__ __noinline__ double gram_schmidt_ordered(double *w, int jb, int m) {
        if constexpr (std::is_same<Team, ClusterTeam>::value) {
            if (local_w) return mgs_ordered(w, jb, m);
        }
        return mgs_ordered_pairs(w, jb, m);
    }

    // The CTA's share of a Krylov vector as up to two runs of doubles: [g0, g0 + n0) and, in the last
    // CTA of a local 1D problem, the boundary moments [g1, g1 + n1).
    __device__ __noinline__ double gram_schmidt(double *w, int jb, int m) {
        const int n = jb + 1, warp = threadIdx.x >> 5, tid = threadIdx.x;
        const long long ldv = P.vstride;
        double *V = vec(4), *ws = nullptr;
        long long g0, g1 = 0;
        int n0, n1 = 0;
        if (std::is_same<Team, ClusterTeam>::value && local_w) {
            const Local1D &L = *reinterpret_cast<const Local1D *>(gs.l1d);
            ws = L.ws;
            g0 = L.e0; n0 = L.l1; g1 = L.eb; n1 = L.ls - L.l1;
        } else {
            const long long np_ = ldv / 2;
            g0 = 2 * (np_ * t.crank / t.ncta);
            n0 = (int)(2 * (np_ * (t.crank + 1) / t.ncta) - g0);
        }
        double *u = ws ? ws - g0 : w;  // w after the first update, by position (run 1: shifted)
        double *u1 = ws ? ws + n0 - g1 : w;
        const bool pair = g0 % 2 == 0 && n0 % 2 == 0 && reinterpret_cast<uintptr_t>(u + g0) % 16 == 0;
        for (int i0 = 0; i0 < n; i0 += 4) {
            double acc[8] = {};
            const double *Ve[4];
            const double2 *Ve2[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                Ve[e] = V + min(i0 + e, jb) * ldv + g0;
                Ve2[e] = RB_CD2(Ve[e]);
            }
            const double *vj = V + jb * ldv;
            if (pair) mgs_dots<double2, 2>(RB_CD2(w + g0), RB_CD2(vj + g0), Ve2, tid, n0 / 2, acc);
            else mgs_dots<double, 4>(w + g0, vj + g0, Ve, tid, n0, acc);
            if (n1 > 0) {
#pragma unroll
                for (int e = 0; e < 4; e++) Ve[e] += g1 - g0;
                mgs_dots<double, 1>(w + g1, vj + g1, Ve, tid, n1, acc);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int e = 0; e < 8; e++) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
            if ((tid & 31) == 0)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (i0 + e < n) gs.red[warp * RB_SM + i0 + e] = acc[e];
                    if (i0 + e < jb) gs.red[warp * RB_SM + n + i0 + e] = acc[4 + e];
                }
        }
        double *h = t.sum_many(gs.red, 2 * n - 1);
        mgs_coefficients(h, n, m);
        double v[1];
        if (pair) v[0] = mgs_update<double2, 2>(RB_CD2(w + g0), RB_D2(u + g0), RB_CD2(V + g0), ldv / 2, tid, n0 / 2, n, h);
        else v[0] = mgs_update<double, 4>(w + g0, u + g0, V + g0, ldv, tid, n0, n, h);
        if (n1 > 0) v[0] += mgs_update<double, 1>(w + g1, u1 + g1, V + g1, ldv, tid, n1, n, h);
        t.template sumk<1>(v);
        const double hn = sqrt(v[0]);
        if (hn > 0.0) {
            const double inv = 1.0 / hn;
            double *Vn = V + n * ldv;
            if (pair) mgs_scale<double2>(RB_CD2(u + g0), RB_D2(Vn + g0), inv, tid, n0 / 2);
            else mgs_scale<double>(u + g0, Vn + g0, inv, tid, n0);
            if (n1 > 0) mgs_scale<double>(u1 + g1, Vn + g1, inv, tid, n1);
        }
        return hn;
    }

    // ---------------------------------------------------------------- gmres(m)
    __device__ __noinline__ SolveStat gmres(double *z, const double *rhs, int restart, int maxit, double tol) {
        const long long N = P.nstate, N2 = P.vstride / 2;  // elements, pairs
        const int m = restart > 1 ? restart : 1;
        SolveStat st = {0, 0.0, 1, CUDART_NAN};
        const double bnorm = sqrt(vdot2(t, rhs, rhs, N2));
        if (bnorm == 0.0) { vzero(t, z, N); return st; }
        double *r = vec(2), *w = vec(3);
        double *H = gs.H;
#define HH(i, j) H[(i) + (m + 1) * (j)]
        int iter = 0, conv = 0;
        double resid = 1.0, resid0 = CUDART_NAN;
        while (iter < maxit && !conv) {
            matvec(r, z); iter++;
            double v1[1] = {0.0};
            {  // r = c − M z
                double2 xc[RB_VU2], xr[RB_VU2];
                const double2 *c2 = RB_CD2(rhs);
                double2 *r2 = RB_D2(r);
                RB_VPAIRS(t, N2, { xc[u_] = c2[q]; xr[u_] = r2[q]; }, {
                    double2 ri;
                    ri.x = xc[u_].x - xr[u_].x;
                    ri.y = xc[u_].y - xr[u_].y;
                    r2[q] = ri;
                    v1[0] += ri.x * ri.x;
                    v1[0] += ri.y * ri.y;
                })
            }
            t.template sumk<1>(v1);
            const double beta = sqrt(v1[0]);
            resid = beta / bnorm;
            if (isnan(resid0)) resid0 = resid;
            if (resid < tol) { conv = 1; break; }
            {
                const double inv = 1.0 / beta;
                double2 *V02 = RB_D2(vec(4));
                const double2 *r2 = RB_CD2(r);
                double2 xr[RB_VU2];
                RB_VPAIRS(t, N2, { xr[u_] = r2[q]; }, { V02[q] = make_double2(xr[u_].x * inv, xr[u_].y * inv); })
            }
            if (t.leader()) {
                for (int i = 0; i <= m; i++) gs.g[i] = 0.0;
                gs.g[0] = beta;
            }
            t.sync();
            int k = 0;
            for (int j = 0; j < m; j++) {
                if (iter >= maxit) break;
                matvec(w, vec(4 + j)); iter++;
                const double hjp1 = P.precision == 1 ? gram_schmidt_ordered(w, j, m) : gram_schmidt(w, j, m);
                if (t.leader()) {
                    HH(j + 1, j) = hjp1;
                    for (int i = 0; i < j; i++) {
                        const double temp = gs.cs[i] * HH(i, j) + gs.sn[i] * HH(i + 1, j);
                        HH(i + 1, j) = -gs.sn[i] * HH(i, j) + gs.cs[i] * HH(i + 1, j);
                        HH(i, j) = temp;
                    }
                    const double denom = hypot(HH(j, j), HH(j + 1, j));
                    if (denom == 0.0) { gs.cs[j] = 1.0; gs.sn[j] = 0.0; }
                    else { gs.cs[j] = HH(j, j) / denom; gs.sn[j] = HH(j + 1, j) / denom; }
                    HH(j, j) = gs.cs[j] * HH(j, j) + gs.sn[j] * HH(j + 1, j);
                    HH(j + 1, j) = 0.0;
                    gs.g[j + 1] = -gs.sn[j] * gs.g[j];
                    gs.g[j] = gs.cs[j] * gs.g[j];
                }
                t.sync();
                k = j + 1;
                resid = fabs(gs.g[j + 1]) / bnorm;
                if (resid < tol) { conv = 1; break; }
                if (hjp1 == 0.0) break;
            }
            if (t.leader()) {
                for (int i = k - 1; i >= 0; i--) {
                    double s = gs.g[i];
                    for (int l = i + 1; l < k; l++) s -= HH(i, l) * gs.y[l];
                    gs.y[i] = HH(i, i) != 0.0 ? s / HH(i, i) : 0.0;
                }
            }
            __syncthreads();
            // z += Σ y_i V_i, in basis order per element
            {
                double2 xz[RB_VU2];
                double2 *z2 = RB_D2(z);
                RB_VPAIRS(t, N2, { xz[u_] = z2[q]; }, {
                    double2 zq = xz[u_];
                    for (int i = 0; i < k; i++) {
                        const double2 v = RB_CD2(vec(4 + i))[q];
                        zq.x += gs.y[i] * v.x;
                        zq.y += gs.y[i] * v.y;
                    }
                    z2[q] = zq;
                })
            }
            t.sync();
            if (conv) break;
        }
#undef HH
        st.iter = iter; st.resid = resid; st.conv = conv; st.rho = rho_estimate(resid0, resid, iter);
        return st;
    }

    // The vector loops of BiCGStab on the grid team: a thread's pairs come by cp.async into its own
    // slots, several turns ahead, so that the reads of the loop's vectors stay in flight while it works
    // (loops that load a batch of pairs and then use it drain the pipe at every turn: 2.6 TB/s at 64³
    // with 256 threads a SM). Same pairs per thread and same order as RB_VPAIRS, so the same sums.
    // f(pair index, x[NV]) for each pair; `local` is free between the phases of a pass.
    template <int NV, class F>
    __device__ __forceinline__ void stream(const double2 *const (&src)[NV], long long N2, F f) {
        const long long q1 = N2 * (t.crank + 1) / t.ncta, q0 = N2 * t.crank / t.ncta + threadIdx.x;
        constexpr int S = NV <= 2 ? 8 : (NV == 3 ? 6 : 4);  // turns in flight
        double2 *slot = reinterpret_cast<double2 *>(local) + threadIdx.x;  // [S][NV][threads]
        auto issue = [&](long long q, int s) {
            if (q < q1)
#pragma unroll
                for (int v = 0; v < NV; v++)
                    cp_zfill<16>(reinterpret_cast<double *>(slot + (s * NV + v) * RB_THREADS),
                                 reinterpret_cast<const double *>(src[v] + q), true);
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll 1
        for (int s = 0; s < S; s++) issue(q0 + s * RB_THREADS, s);
        int s = 0;
#pragma unroll 1
        for (long long q = q0; q < q1; q += RB_THREADS) {
            asm volatile("cp.async.wait_group %0;" ::"n"(S - 1) : "memory");
            double2 x[NV];
#pragma unroll
            for (int v = 0; v < NV; v++) x[v] = slot[(s * NV + v) * RB_THREADS];
            issue(q + S * RB_THREADS, s);
            s = s + 1 == S ? 0 : s + 1;
            f(q, x);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    static constexpr long long stream_bytes = 20LL * RB_THREADS * 16;  // the largest S·NV
    template <int NV, class F>
    __device__ __forceinline__ void vloop(const double2 *const (&src)[NV], long long N2, F f) {
        if constexpr (std::is_same<Team, GridTeam>::value) {
            if (local_bytes >= stream_bytes) {
                stream<NV>(src, N2, f);
                return;
            }
        }
        double2 xv[4][NV];
        RB_VPAIRS_D(t, N2, 4, {
#pragma unroll
            for (int v = 0; v < NV; v++) xv[u_][v] = src[v][q];
        }, { f(q, xv[u_]); })
    }

    // ---------------------------------------------------------------- bicgstab
    // Vector loops over 16-byte element pairs of CTA-contiguous slices (the pad element of an odd
    // state stays zero in every vector).
    __device__ __noinline__ SolveStat bicgstab(double *z, const double *rhs, int maxit, double tol) {
        const long long N = P.nstate, N2 = P.vstride / 2;
        SolveStat st = {0, 0.0, 1, CUDART_NAN};
        const double bnorm = sqrt(vdot2(t, rhs, rhs, N2));
        if (bnorm == 0.0) { vzero(t, z, N); return st; }
        double *r = vec(2), *rh = vec(3), *p = vec(4), *v = vec(5), *s = vec(6), *tt = vec(7);
        double2 *r2 = RB_D2(r), *rh2 = RB_D2(rh), *p2 = RB_D2(p), *v2 = RB_D2(v), *s2 = RB_D2(s), *z2 = RB_D2(z);
        const double2 *c2 = RB_CD2(rhs), *t2 = RB_CD2(tt);
        const double2 zero2 = make_double2(0.0, 0.0);
        matvec(r, z);
        double a1[1] = {0.0};
        vloop<2>({c2, r2}, N2, [&](long long q, const double2 (&x)[2]) {
            const double2 ri = make_double2(x[0].x - x[1].x, x[0].y - x[1].y);
            r2[q] = ri; rh2[q] = ri; p2[q] = zero2; v2[q] = zero2;
            a1[0] += ri.x * ri.x;
            a1[0] += ri.y * ri.y;
        });
        t.template sumk<1>(a1);
        int iter = 1, conv = 0;
        double resid = sqrt(a1[0]) / bnorm, resid0 = resid;
        if (resid < tol) { st.iter = iter; st.resid = resid; st.conv = 1; st.rho = CUDART_NAN; return st; }
        double rho_old = 1.0, alpha = 1.0, omega = 1.0;
        const double tiny = 1e-300;
        // (r̂·r) of the coming iteration: the initial loop's Σ r² (r̂ = r there), then the last
        // loop's second sum (the same terms, in the same order per thread, as a separate dot)
        double rho_next = a1[0];
        while (iter < maxit) {
            const double rho_new = rho_next;
            if (fabs(rho_new) < tiny) break;
            const double beta = (rho_new / rho_old) * (alpha / omega);
            vloop<3>({r2, p2, v2}, N2, [&](long long q, const double2 (&x)[3]) {
                p2[q] = make_double2(x[0].x + 1.0 * (beta * (x[1].x + (-omega) * x[2].x)),
                                     x[0].y + 1.0 * (beta * (x[1].y + (-omega) * x[2].y)));
            });
            t.sync();
            matvec(v, p); iter++;
            double a0[1] = {0.0};
            vloop<2>({rh2, v2}, N2, [&](long long, const double2 (&x)[2]) {
                a0[0] += x[0].x * x[1].x;
                a0[0] += x[0].y * x[1].y;
            });
            t.template sumk<1>(a0);
            const double denom = a0[0];
            if (fabs(denom) < tiny) break;
            alpha = rho_new / denom;
            double a2[1] = {0.0};
            vloop<2>({r2, v2}, N2, [&](long long q, const double2 (&x)[2]) {
                const double2 si = make_double2(x[0].x + (-alpha) * x[1].x, x[0].y + (-alpha) * x[1].y);
                s2[q] = si;
                a2[0] += si.x * si.x;
                a2[0] += si.y * si.y;
            });
            t.template sumk<1>(a2);
            const double sn_ = sqrt(a2[0]);
            if (sn_ / bnorm < tol) {
                vaxpy(t, alpha, p, z, N);
                resid = sn_ / bnorm;
                conv = 1;
                break;
            }
            matvec(tt, s); iter++;
            double a3[2] = {0.0, 0.0};
            vloop<2>({t2, s2}, N2, [&](long long, const double2 (&x)[2]) {
                a3[0] += x[0].x * x[0].x;
                a3[0] += x[0].y * x[0].y;
                a3[1] += x[0].x * x[1].x;
                a3[1] += x[0].y * x[1].y;
            });
            t.template sumk<2>(a3);
            if (a3[0] < tiny) break;
            omega = a3[1] / a3[0];
            double a4[2] = {0.0, 0.0};
            vloop<5>({z2, p2, s2, t2, rh2}, N2, [&](long long q, const double2 (&x)[5]) {
                z2[q] = make_double2((x[0].x + alpha * x[1].x) + omega * x[2].x, (x[0].y + alpha * x[1].y) + omega * x[2].y);
                const double2 ri = make_double2(x[2].x + (-omega) * x[3].x, x[2].y + (-omega) * x[3].y);
                r2[q] = ri;
                a4[0] += ri.x * ri.x;
                a4[0] += ri.y * ri.y;
                a4[1] += x[4].x * ri.x;
                a4[1] += x[4].y * ri.y;
            });
            t.template sumk<2>(a4);
            rho_next = a4[1];
            resid = sqrt(a4[0]) / bnorm;
            if (resid < tol) { conv = 1; break; }
            if (fabs(omega) < tiny) break;
            rho_old = rho_new;
        }
        st.iter = iter; st.resid = resid; st.conv = conv; st.rho = rho_estimate(resid0, resid, iter);
        return st;
    }

    // ---------------------------------------------------------------- sn_one_speed
    __device__ __noinline__ SolveStat one_speed(double *flux_g) {
        const long long N = P.nstate, nphi = P.nphi;
        const long long nE = (long long)P.nd * P.nm4 * P.ncell;
        // zero-source short-circuit (sn_one_speed.jl:115-120)
        int any = 0;
        for (int f = 0; f < 2 * P.ndims; f++) {
            const double *src = P.surf[f];
            if (!src) continue;
            for (long long k = t.rank(); k < (long long)P.np_source * P.fcells[f / 2]; k += t.size())
                if (src[ig + (long long)P.ng * k] != 0.0) any = 1;
        }
        for (long long i = t.rank(); i < nphi; i += t.size()) if (P.qlout[i] != 0.0) any = 1;
        if (P.csd) for (long long i = t.rank(); i < nE; i += t.size()) if (phiE_in[i] != 0.0) any = 1;
        any = t.any(any);
        if (!any) {
            for (long long i = t.rank(); i < nphi; i += t.size()) flux_g[i] = 0.0;
            if (P.csd) for (long long i = t.rank(); i < nE; i += t.size()) phiE_out[i] = 0.0;
            t.sync();
            SolveStat s = {1, 0.0, 1, CUDART_NAN};
            return s;
        }
        double *z = vec(0);
        vzero(t, z, N);  // initial state: 𝚽l of the group = 0, boundary in-moments = 0
        SolveStat st;
        const bool mixed = P.precision == 1;
        if (P.accel == 0 || P.accel == 1) {
            st = livolant(z, P.maxit, mixed ? fmax(P.tol, RB_MIXED_TOL) : P.tol, P.accel == 0 ? 0 : 3);
        } else if (P.accel == 2) {
            st = anderson(z, P.depth, P.maxit, mixed ? fmax(P.tol, RB_MIXED_TOL) : P.tol);
        } else {
            double *rhs = vec(1);
            pass(z, rhs, 0, 0, 1);  // c = T(0), FP64 in both forms
            // The mixed form solves with the FP32 operator to RB_MIXED_TOL1, then takes one outer
            // defect-correction step: the residual r = c − (I − A)·z with the FP64 operator, the
            // correction δ from the FP32-operator solve of (I − A)·δ = r to the tolerance that
            // brings the whole residual to `tol`, z ← z + δ.
            const double tol1 = mixed ? fmax(P.tol, RB_MIXED_TOL1) : P.tol;
            if (P.accel == 3) st = gmres(z, rhs, P.restart, P.maxit, tol1);
            else st = bicgstab(z, rhs, P.maxit, tol1);
            if (mixed) {
                double *dz = vec(P.nvec - 2), *res = vec(P.nvec - 1);
                pass(z, res, 1, 1, 1);  // res = z − A·z, FP64
                double v[2] = {0.0, 0.0};
                for (long long i = t.rank(); i < N; i += t.size()) {
                    const double ri = rhs[i] - res[i];
                    res[i] = ri;
                    v[0] += ri * ri;
                    v[1] += rhs[i] * rhs[i];
                }
                t.template sumk<2>(v);
                const double rel = v[1] > 0.0 ? sqrt(v[0] / v[1]) : 0.0;
                if (rel >= P.tol) {
                    vzero(t, dz, N);
                    const double tol2 = fmax(P.tol / rel, RB_MIXED_TOL);
                    SolveStat s2;
                    if (P.accel == 3) s2 = gmres(dz, res, P.restart, P.maxit, tol2);
                    else s2 = bicgstab(dz, res, P.maxit, tol2);
                    vaxpy(t, 1.0, dz, z, N);
                    st.iter += s2.iter + 1;
                    st.resid = s2.resid * rel;
                    st.conv = s2.conv;
                } else {
                    st.iter += 1;
                    st.resid = rel;
                    st.conv = 1;
                }
            }
        }
        // reconstruction pass (sn_one_speed.jl:184-187)
        double *out = vec(1);
        pass(z, out, 0, 0, 1, 1);
        vcopy(t, flux_g, out, nphi);
        return st;
    }
};

// ------------------------------------------------------------------------------------------
// the group loop of compute_flux(::SN) for one problem (sn_flux.jl:146-224)
// ------------------------------------------------------------------------------------------
template <class Team, bool LO = false>
__device__ void solve_problem(Team &t, const DevProblem &P0, GroupShared &gs, void *local = nullptr,
                              long long local_bytes = 0) {
    if (threadIdx.x == 0) gs.prob = P0;
    __syncthreads();
    const DevProblem &P = gs.prob;
    const int local_ok = (local && local1d_ok(P, (int)t.ncta, local_bytes)) ? 1 : 0;
    const int local_w = (local && local1d_w(P, (int)t.ncta, local_bytes)) ? 1 : 0;
    const int ng = P.ng, nmat = P.nmat, np = P.np, nd = P.nd, nm = P.nm5;
    const long long nphi = P.nphi, ncell = P.ncell;
    const long long nE = (long long)nd * P.nm4 * ncell;
    const int st_ = P.solver_type;
    double *phiE_in = P.phiE_a, *phiE_out = P.phiE_b;
    // the pad element of each Krylov vector (odd nstate) starts and stays zero
    if (P.vstride > P.nstate)
        for (int k = t.rank(); k < P.nvec; k += t.size()) P.vecs[(long long)k * P.vstride + P.nstate] = 0.0;
    if (P.csd) { vzero(t, phiE_in, nE); vzero(t, phiE_out, nE); }
    // the octant sweep's progress flags count up from zero within this solve
    if (P.ndims == 3)
        for (int k = t.rank(); k < RB_OCT_MAXCTA; k += t.size()) P.oct_flags[k] = 0ull;
    if (threadIdx.x == 0) gs.oct_epoch = 0;
    if constexpr (std::is_same<Team, ClusterTeam>::value) {
        if (LO || local_ok) {
            Local1D &L = *reinterpret_cast<Local1D *>(gs.l1d);
            if (threadIdx.x == 0) L = Local1D(P, t.crank, t.ncta, local, local_bytes);
            __syncthreads();
            local1d_load_ops(P, L);
        }
    }
    t.sync();
    long long npass = 0;
    for (int ig = 0; ig < ng; ig++) {
        // per-group constants, one copy per CTA
        for (int m = threadIdx.x; m < nmat; m += blockDim.x) {
            gs.sigt[m] = P.sigma_t[ig + (long long)ng * m];
            if (P.csd) {
                const double dE = P.e_width[ig];
                gs.sm[m] = P.s_minus[ig + (long long)ng * m] / dE;
                gs.sp[m] = P.s_plus[ig + (long long)ng * m] / dE;
            } else {
                gs.sm[m] = gs.sp[m] = 0.0;
            }
            gs.tg[m] = (st_ == 2 || st_ == 4) ? P.t_mom[ig + (long long)ng * m] : 0.0;
        }
        __syncthreads();
        if (P.csd) {  // CSD block of the cell matrix: Σ_w (S_w/ΔE)·K_w + (S⁺/ΔE)·B
            const int nn = nm * nm;
            for (long long o = t.rank(); o < (long long)nmat * nn; o += t.size()) {
                const int m = (int)(o / nn), e = (int)(o % nn);
                const double dE = P.e_width[ig];
                double v = gs.sp[m] * P.Bcsd[e];
                for (int w = 0; w < P.oE; w++)
                    v += (P.s_mom[ig + (long long)ng * (m + (long long)nmat * w)] / dE) * P.Kcsd[(long long)w * nn + e];
                P.scsd[o] = v;
            }
        }
        // ys[m][p] = Σs_in[m, pl[p]]: the in-group scattering source of moment p (zero for the
        // solvers without it, sn_inner_pass.jl:21); T[m] scales the Fokker-Planck product
        const bool scat = (st_ != 4 && st_ != 5 && st_ != 6);
        for (long long o = t.rank(); o < (long long)nmat * np; o += t.size()) {
            const int p = (int)(o % np);
            const int m = (int)(o / np);
            P.kmat[o] = scat ? P.sigma_s[m + (long long)nmat * (ig + (long long)ng * (ig + (long long)ng * P.pl[p]))] : 0.0;
        }
        // Qlout = Σ_{gi≠ig} Σs[mat,gi,ig,l]·𝚽[gi] + volume source (scattering_source.jl:59-68;
        // groups above ig are still zero in the single outer iteration, sn_flux.jl:150,157)
        for (long long o = t.rank(); o < nphi; o += t.size()) {
            const int p = (int)(o % np);
            const long long c = o / ((long long)np * nm);
            const int m = P.mat[c];
            double q = 0.0;
            if (st_ != 4 && st_ != 5) {
                const double *ss = P.sigma_s + m + (long long)nmat * (long long)ng * (ig + (long long)ng * P.pl[p]);
                for (int gi = 0; gi < ig; gi++) q += ss[(long long)nmat * gi] * P.flux[(long long)gi * nphi + o];
            }
            // the volume source: particle source + fixed source (transport.jl:89-90)
            if (P.pvol || P.vol) {
                double vs = P.pvol ? P.pvol[(long long)ig * nphi + o] : 0.0;
                if (P.vol) vs = vs + P.vol[(long long)ig * nphi + o];
                q += vs;
            }
            P.qlout[o] = q;
        }
        if (P.csd && ig != 0) {  // 𝚽E12 .* ΔE[ig] / ΔE[ig-1]
            const double r1 = P.e_width[ig], r0 = P.e_width[ig - 1];
            for (long long i = t.rank(); i < nE; i += t.size()) phiE_in[i] = phiE_in[i] * r1 / r0;
        }
        t.sync();
        if constexpr (std::is_same<Team, ClusterTeam>::value) {
            if (LO || local_ok) {
                Local1D &L = *reinterpret_cast<Local1D *>(gs.l1d);
                local1d_group_setup(P, L);
                local1d_factor_fixed(P, gs, L);
            }
        }
        // Qnout = Mn·Qlout, kept for the passes of this group. The local 1D pass holds its region:
        // the product stages in GroupShared there.
        {
            const bool own = local != nullptr && !(LO || local_ok);
            m2d_tiles(t, P, gs, own ? local : (void *)gs.tile, own ? local_bytes : (long long)sizeof(gs.tile), P.qlout,
                      nullptr, P.qnout, 0);
        }
        t.sync();
        Solver<Team, LO> S{t, P, gs, ig, phiE_in, phiE_out, 0};
        S.local = local;
        S.local_bytes = local ? local_bytes : 0;
        S.local_ok = local_ok;
        S.local_w = local_w;
        SolveStat s = S.one_speed(P.flux + (long long)ig * nphi);
        npass += S.npass;
        if (t.rank() == 0) {
            P.rho[ig] = s.rho; P.resid[ig] = s.resid; P.iters[ig] = s.iter; P.conv[ig] = s.conv;
            if (!s.conv) atomicOr(P.status, RB_DEV_NOT_CONVERGED);
        }
        double *tmp = phiE_in; phiE_in = phiE_out; phiE_out = tmp;
        t.sync();
    }
    // 𝚽cutoff[p,is,c] = Σ_n Dn[p,n]·𝚽E12[n,is,c] for is < Nm4 (sn_flux.jl:215-218)
    if (P.csd) {
        for (long long o = t.rank(); o < nphi; o += t.size()) {
            const int p = (int)(o % np);
            const int is = (int)((o / np) % nm);
            const long long c = o / ((long long)np * nm);
            double s = 0.0;
            if (is < P.nm4)
                for (int n = 0; n < nd; n++)
                    s += P.dn[p + (long long)np * n] * phiE_in[n * P.pe_sn + (is + (long long)P.nm4 * c) * P.psi_sc];
            P.cutoff[o] = s;
        }
    }
    if (t.rank() == 0) *P.passes = npass;
    t.sync();
}

// ------------------------------------------------------------------------------------------
// the persistent kernels (each defined in its own translation unit, rb_kernel_*.cu)
// ------------------------------------------------------------------------------------------
// Dynamic shared memory: GroupShared, then `local_bytes` for the local 1D pass (and the 3D
// octant sweep). Clusters pull problems from the work queue `queue`.
__global__ void __launch_bounds__(RB_THREADS, 1) solve_batch_kernel(DevProblem *const *probs, int nprob, int *queue,
                                                                 int local_bytes);
// The same loop for batches whose every problem takes the local 1D pass: the kernel carries no
// other pass, so its registers go to that path alone.
__global__ void __launch_bounds__(RB_THREADS, 1) solve_local1d_kernel(DevProblem *const *probs, int nprob, int *queue,
                                                                   int local_bytes);
// One large (2D/3D) problem on the whole GPU: a cooperative launch, one team of every CTA.
__global__ void __launch_bounds__(RB_THREADS, 1) solve_grid_kernel(DevProblem *prob, double *gpart, int local_bytes);

}  // namespace rb
