// rb_product.cuh -- the FP64 moment<->direction products on the FP64 tensor pipe (mma.sync
// m8n8k4.f64: tcgen05 has no FP64 kind, and the FP64 pipe behind mma.sync is the only one at the
// full 37 TFLOP/s measured on a B200).
//
// The products are the M2D and D2M lines of sn_sweep_{1,2,3}D.jl (Qn = Mn[n,:]·Ql,
// 𝚽l += Dn[:,n]·𝚽n) with the in-group scattering (scattering_source.jl:25-30) and Fokker-Planck
// (fokker_planck_source.jl:29-33) sources folded in:
//   out[col, i] = pre[col, i] + alpha·Σ_k (s(k, col)·A[i, k] + t(col)·B[i, k])·X[col, k]
// A column ("col") is one cell moment of one cell; its values are contiguous in memory, or (the
// angular arrays of one-moment 2D problems) those of neighbouring columns are.
//
// Split. The columns are the M side of the MMA (8 per tile) and the operator's rows the N side, so
// a lane reads its column's run of k as it lies in memory (4 lanes = one 32-byte sector, or 8
// columns = two) straight into registers, a chunk of 16 or 32 k ahead, and writes two neighbouring outputs (a quad = 64 bytes of
// a column). Only the operator is staged in shared memory, once per call, k-major with a row of
// 8·NT + 4 doubles (the 4×4 block of a half-warp then falls into 16 different banks). No block
// barrier stands between the column tiles of a call: a warp runs through its own.
// An operator too large for the region is cut by rows over the CTAs of the team (CTA r takes row
// block r mod nrb), which reads the columns nrb times but never reloads the operator.
//
// What bounds it: the 3D products stream z and ψ (HBM and L2), the 2D ones with their 168
// directions the FP64 pipe, the 1D ones the latency of a call. M2D of 48×41×35 cells, S8, two parts:
// 350 us as staged panels on the FP64 cores, 116 here; 128×128, S12: 203 and 90; 152 columns of a
// slab team, 32 rows, two parts: 35 and 14.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace rb {

struct Prod64 {
    const double *A, *B;  // operator parts [i·ldi + lda·k], i < ni, k < nk (B may be null)
    int lda, ldi, ni, nk;
    const double *X;      // [k·sx + ldx·col]
    long long sx, ldx, ncol;
    const double *ks;     // scale of part A: ks[m·ksld + k], m = mat[col / nm]
    int ksld;
    const double *tg;     // scale of part B: tg[m] (of part A when ks and B are null); null: 1
    const int *mat;
    int nm;
    const double *pre;    // added term, laid out as out (null: 0)
    double alpha;
    double *out;          // [i·so + col·ldo]
    long long so, ldo;
    // half of the directions only: those n whose (sel[n] >= 0) is selpos. selk: n is k (the others'
    // operator columns and values of X are taken as zero, whatever X holds there); else n is i (the
    // others' outputs are left alone). null: all.
    const double *sel = nullptr;
    bool selk = false, selpos = false;
    // both parts on a piece of k before the next piece (the columns are loaded once, not twice): the
    // plain form. The mixed form, whose FP32 roundings follow the last bit, keeps part A before B.
    bool interleave = false;
};

#define RB_PROD_MAXNT 12  // row tiles (of 8) a warp accumulates at once

__host__ __device__ __forceinline__ int prod_kp(int nk) { return (nk + 3) & ~3; }
// row tiles are instantiated in even counts
__host__ __device__ __forceinline__ int prod_nt(int ni) { return ((ni + 7) / 8 + 1) & ~1; }
// bytes of an operator block of nt row tiles
__host__ __device__ __forceinline__ long long prod_bytes(int nt, int nk, int parts) {
    return (long long)parts * prod_kp(nk) * (8 * nt + 4) * 8;
}
// row blocks of an operator: the fewest whose block has at most RB_PROD_MAXNT tiles and fits in
// `bytes`; 0 when no block of two tiles does
__host__ __device__ __forceinline__ int prod_blocks(int ni, int nk, int parts, long long bytes) {
    const int t = (ni + 7) / 8;
    for (int nrb = (t + RB_PROD_MAXNT - 1) / RB_PROD_MAXNT;; nrb++) {
        const int nt = prod_nt(8 * ((t + nrb - 1) / nrb));
        if (prod_bytes(nt, nk, parts) <= bytes) return nrb;
        if (nt <= 2) return 0;
    }
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
__device__ __forceinline__ double lds64(uint32_t a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}

__device__ __forceinline__ int lds32(uint32_t a) {
    int v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// asynchronous copy global -> shared of B bytes, zeros instead where `in` is false
template <int B>
__device__ __forceinline__ void cp_zfill(double *dst, const double *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(B), "r"(in ? B : 0)
                 : "memory");
}

// Rows [i0, i0 + 8·nt) of the operator into shared memory, zero beyond ni and nk: every copy in
// flight at once (a row per warp, 16 bytes a lane where the operator's rows are aligned). selk: the
// first word of a row's padding says whether its k is in.
__device__ __forceinline__ void prod_load_op(const Prod64 &a, double *op, int i0, int nt) {
    const int kp = prod_kp(a.nk), ld = 8 * nt + 4, parts = a.B ? 2 : 1;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const bool vec = a.ldi == 1 && a.lda % 2 == 0 && i0 % 2 == 0 && a.ni % 2 == 0 && reinterpret_cast<uintptr_t>(a.A) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(a.B) % 16 == 0;
    for (int r = threadIdx.x >> 5; r < parts * kp; r += nw) {
        const bool pb = r >= kp;
        const int k = pb ? r - kp : r;
        const double *src = (pb ? a.B : a.A) + (k < a.nk ? (long long)a.lda * k : 0);
        const bool kin = k < a.nk && !(a.sel && a.selk && (a.sel[k] >= 0.0) != a.selpos);
        if (a.selk && lane == 0) *reinterpret_cast<int *>(op + r * ld + 8 * nt) = kin;
        if (vec) {
            for (int i = 2 * lane; i < 8 * nt; i += 64) {
                const bool in = kin && i0 + i < a.ni;
                cp_zfill<16>(op + r * ld + i, in ? src + i0 + i : src, in);
            }
        } else {
            for (int i = lane; i < 8 * nt; i += 32) {
                const bool in = kin && i0 + i < a.ni;
                cp_zfill<8>(op + r * ld + i, in ? src + (long long)(i0 + i) * a.ldi : src, in);
            }
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The column tiles w0, w0 + wstep, … (groups of MT tiles of 8) against the resident operator block.
// With a.selk a column in which the directions left out hold an infinity or NaN comes out non-finite (zero
// operator columns times it): such a group is not stored, and the result is true; prod_run then calls the
// SELK variant, which takes those directions' values as zero by the flags of the operator's rows. A look at
// the sums is thus all that ordinary columns pay (the flags in every product: 128×128, S12 4 %; in the
// boundary products alone, whose code then is not the M2D and D2M products': 41×30, S6, four moments and
// 48×41×35, S8 electrons 2 %; a call of the SELK variant from here: 128×128, S12 11 %, by its registers).
template <int NT, int MT, bool SELK>
__device__ __noinline__ bool prod_tiles(const Prod64 &a_, const double *op, int i0, int w0, int wstep) {
    const Prod64 a = a_;
    const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    constexpr int LD = 8 * NT + 4;
    constexpr int CH = NT * MT >= 16 ? 4 : 8;  // k-steps (of 4) of a column loaded ahead, by the registers left
    // one accumulator takes the terms in the order of a plain loop over k (the MMA itself adds its
    // four products in order, each rounded: an FMA chain), through part A, then part B, or piece by
    // piece of both
    const int kp = prod_kp(a.nk), nks = kp / 4, npc = (nks + CH - 1) / CH;
    const bool two = a.B != nullptr;
    const bool inter = two && a.interleave;
    const int nch = two && !inter ? 2 * npc : npc;
    const uint32_t ob = (uint32_t)__cvta_generic_to_shared(op) + (uint32_t)(q * LD + r) * 8;
    const long long ngrp = (a.ncol + 8 * MT - 1) / (8 * MT);
    if (w0 >= ngrp) return false;
    bool bad = false;
    const bool rows = a.sel && !a.selk;
    const bool vec = !rows && a.so == 1 && (a.ldo % 2 == 0) && (reinterpret_cast<uintptr_t>(a.out) % 16 == 0) &&
                     (reinterpret_cast<uintptr_t>(a.pre) % 16 == 0);
    double xn[MT][CH];
    auto load = [&](long long g, int ch) {
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            const long long col = (g * MT + mt) * 8 + r;
            const double *xp = a.X + (col < a.ncol ? col : 0) * a.ldx;
#pragma unroll
            for (int u = 0; u < CH; u++) {
                const int k = ((ch < npc ? ch : ch - npc) * CH + u) * 4 + q;
                xn[mt][u] = (k < a.nk && col < a.ncol) ? xp[k * a.sx] : 0.0;
            }
        }
    };
    load(w0, 0);
    for (long long g = w0; g < ngrp; g += wstep) {
        double acc[MT][NT][2];
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
            for (int n = 0; n < NT; n++) acc[mt][n][0] = acc[mt][n][1] = 0.0;
        const double *kq[MT];
        double tq[MT];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            kq[mt] = nullptr;
            tq[mt] = 1.0;
            const long long col = (g * MT + mt) * 8 + r;
            if ((a.ks || a.tg) && col < a.ncol) {
                const int m = a.mat[a.nm == 1 ? col : (long long)((unsigned)col / (unsigned)a.nm)];
                if (a.ks) kq[mt] = a.ks + (long long)m * a.ksld;
                if (a.tg) tq[mt] = a.tg[m];
            }
        }
        for (int ch = 0; ch < nch; ch++) {
            const bool pb = ch >= npc;
            const int c0 = (pb ? ch - npc : ch) * CH;
            double xc[MT][CH], sc[MT][CH];
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int u = 0; u < CH; u++) {
                    xc[mt][u] = xn[mt][u];
                    const int k = (c0 + u) * 4 + q;
                    sc[mt][u] = (kq[mt] && !pb) ? (k < a.nk ? kq[mt][k] : 0.0) : ((two && !pb) ? 1.0 : tq[mt]);
                }
            if (ch + 1 < nch) load(g, ch + 1);
            else if (g + wstep < ngrp) load(g + wstep, 0);
#pragma unroll
            for (int u = 0; u < CH; u++) {
                const int ks = c0 + u;
                if (ks < nks) {
                    double av[MT];
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) av[mt] = sc[mt][u] * xc[mt][u];
                    const uint32_t o = ob + (uint32_t)(ks * 4 + (pb ? kp : 0)) * (LD * 8);
                    if constexpr (SELK) {
                        const bool in = lds32(o + (uint32_t)(8 * NT - r) * 8) != 0;
#pragma unroll
                        for (int mt = 0; mt < MT; mt++) av[mt] = in ? av[mt] : 0.0;
                    }
#pragma unroll
                    for (int n = 0; n < NT; n++) {
                        const double b = lds64(o + n * 64);
#pragma unroll
                        for (int mt = 0; mt < MT; mt++) dmma(acc[mt][n], av[mt], b);
                    }
                    if (inter) {
#pragma unroll
                        for (int mt = 0; mt < MT; mt++) av[mt] = tq[mt] * xc[mt][u];
#pragma unroll
                        for (int n = 0; n < NT; n++) {
                            const double b = lds64(o + (uint32_t)kp * (LD * 8) + n * 64);
#pragma unroll
                            for (int mt = 0; mt < MT; mt++) dmma(acc[mt][n], av[mt], b);
                        }
                    }
                }
            }
        }
        if (!SELK && a.selk) {
            int most = 0;
#pragma unroll
            for (int mt = 0; mt < MT; mt++)
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int e = 0; e < 2; e++) most = max(most, __double2hiint(acc[mt][n][e]) & 0x7fffffff);
            if (__any_sync(0xffffffffu, most >= 0x7ff00000)) {
                bad = true;
                continue;
            }
        }
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            const long long col = (g * MT + mt) * 8 + r;
            if (col >= a.ncol) continue;
            const long long o0 = col * a.ldo + (i0 + 2 * q) * a.so;
            if (vec) {
                double2 pv[NT];
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const int i = i0 + 8 * n + 2 * q;
                    pv[n] = make_double2(0.0, 0.0);
                    if (a.pre) {
                        if (i + 1 < a.ni) pv[n] = *reinterpret_cast<const double2 *>(a.pre + o0 + 8 * n);
                        else if (i < a.ni) pv[n].x = a.pre[o0 + 8 * n];
                    }
                }
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const int i = i0 + 8 * n + 2 * q;
                    const double2 v = make_double2(fma(a.alpha, acc[mt][n][0], pv[n].x), fma(a.alpha, acc[mt][n][1], pv[n].y));
                    if (i + 1 < a.ni) *reinterpret_cast<double2 *>(a.out + o0 + 8 * n) = v;
                    else if (i < a.ni) a.out[o0 + 8 * n] = v.x;
                }
            } else {
                double pv[NT][2];
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int e = 0; e < 2; e++)
                        pv[n][e] = (a.pre && i0 + 8 * n + 2 * q + e < a.ni) ? a.pre[o0 + (8 * n + e) * a.so] : 0.0;
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int e = 0; e < 2; e++)
                        if (i0 + 8 * n + 2 * q + e < a.ni && !(rows && (a.sel[i0 + 8 * n + 2 * q + e] >= 0.0) != a.selpos))
                            a.out[o0 + (8 * n + e) * a.so] = fma(a.alpha, acc[mt][n][e], pv[n][e]);
            }
        }
    }
    return bad;
}

// Dispatch on the row tiles of the block; pairs of column tiles per warp (half the operator reads)
// where every warp still gets one. Sums added to the outputs of earlier ones (a cut along k) cannot be
// computed twice and take the flags at once.
__device__ __forceinline__ void prod_run(const Prod64 &a, const double *op, int i0, int nt, int w0, int wstep) {
    const bool pair = a.ncol >= 16LL * wstep, flags = a.selk && a.pre == a.out;
#define RB_PROD_CASE(NT_)                                                  \
    case NT_:                                                              \
        if (pair) {                                                        \
            if (flags || prod_tiles<NT_, 2, false>(a, op, i0, w0, wstep))  \
                prod_tiles<NT_, 2, true>(a, op, i0, w0, wstep);            \
        } else {                                                           \
            if (flags || prod_tiles<NT_, 1, false>(a, op, i0, w0, wstep))  \
                prod_tiles<NT_, 1, true>(a, op, i0, w0, wstep);            \
        }                                                                  \
        break;
    switch (nt) {
        RB_PROD_CASE(2)
        RB_PROD_CASE(4)
        RB_PROD_CASE(6)
        RB_PROD_CASE(8)
        RB_PROD_CASE(10)
        RB_PROD_CASE(12)
    }
#undef RB_PROD_CASE
}

// The product of a team: row blocks and column tiles dealt to its CTAs, the operator block in
// `region`. An operator whose smallest row block does not fit is cut along k, each cut added to
// the outputs of the ones before it (a column stays with its warp, so no barrier orders them).
template <class Team>
__device__ void prod64_team(const Team &t, const Prod64 &a0, void *region, long long bytes) {
    double *op = reinterpret_cast<double *>(region);
    const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5;
    Prod64 a = a0;
    int nparts = 1, nseg = 1, parts = a.B ? 2 : 1;
    int nrb = prod_blocks(a.ni, a.nk, parts, bytes);
    if (nrb > 0) {  // few columns: more row blocks (of at least two tiles), so that every warp has a task
        const long long tasks = (a.ncol + 7) / 8, warps = (long long)t.ncta * nw;
        const int most = ((a.ni + 7) / 8 + 1) / 2;
        if (tasks * nrb < warps) nrb = max(nrb, min(most, (int)(warps / tasks)));
    }
    if (nrb == 0) {  // one part at a time, its k in pieces that fit
        nparts = parts;
        parts = 1;
        while ((nrb = prod_blocks(a.ni, (a0.nk + nseg - 1) / nseg, 1, bytes)) == 0) nseg++;
    }
    const int seg = (a0.nk + nseg - 1) / nseg;
    const int tiles = (a.ni + 7) / 8, per = (tiles + nrb - 1) / nrb, nt = prod_nt(8 * per);
    const int npar = nrb < (int)t.ncta ? nrb : (int)t.ncta;  // row blocks in parallel
    const int ngrp = (int)t.ncta / npar;                     // CTAs of a row block
    if ((int)t.crank < npar * ngrp)
        for (int b = (int)t.crank % npar; b < nrb && 8 * per * b < a0.ni; b += npar)
            for (int part = 0; part < nparts; part++)
                for (int sg = 0; sg < nseg; sg++) {
                    if (nparts * nseg > 1) {
                        const int k0 = sg * seg;
                        a.nk = min(seg, a0.nk - k0);
                        a.A = (part ? a0.B : a0.A) + (long long)a.lda * k0;
                        a.B = nullptr;
                        a.X = a0.X + k0 * a.sx;
                        if (a0.selk && a0.sel) a.sel = a0.sel + k0;
                        a.ks = (part || !a0.ks) ? nullptr : a0.ks + k0;
                        a.tg = part ? a0.tg : nullptr;
                        a.pre = part + sg > 0 ? a0.out : a0.pre;
                    }
                    a.ni = min(a0.ni, 8 * per * (b + 1));
                    __syncthreads();
                    prod_load_op(a, op, 8 * per * b, nt);
                    __syncthreads();
                    prod_run(a, op, 8 * per * b, nt, ((int)t.crank / npar) * nw + warp, ngrp * nw);
                }
    __syncthreads();
}

}  // namespace rb
