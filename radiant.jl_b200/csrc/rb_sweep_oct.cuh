// rb_sweep_oct.cuh -- 2D and 3D sweeps of one-moment cells (order-1 closures in every axis and
// in energy: the diamond-difference / DG0 cells of sn_2D_bte.jl:35-116, sn_2D_bfp.jl:45-154,
// sn_3D_bte.jl:42-152, sn_3D_bfp.jl:52-191), in FP64 (plain form) or FP32 (mixed form).
//
// 3D: directions are held grouped by octant, and all directions of one octant share one sweep
// order, so a thread owns one x-pencil (iy, iz) of a TY×TZ tile and solves up to DB directions
// of one octant at each cell it visits. Inside a tile the pencils form a hyperplane wavefront:
// at local step σ the pencil (jy, jz) solves column σ − jy − jz. The x face stays in registers;
// the y face of the pencil below comes by warp shuffle (it is the neighbouring lane); the z face
// of the pencil behind comes through shared memory, double-buffered by step parity. Tiles hand
// their outgoing y/z faces to the downstream tiles through per-direction face planes in global
// memory. Every (octant batch, tile) is one task on one CTA of the team; a tile is paced by its
// upwind tiles through per-CTA progress flags (a release after each pair of steps, an acquire
// before the faces of a step are staged), so it runs about one tile height behind them with no
// team barrier inside the sweep. A step's cells are staged a step ahead with cp.async, each warp
// its own 32 cells, and written back by the same lanes.
// Each cell sees the same upwind faces as in the reference's lexicographic order
// (sn_sweep_3D.jl:73-110), so the result equals it up to rounding.
//
// 2D: the KBA wavefront of sweep_md (rows of a direction skewed by one column per row), a warp on 32
// rows of a direction: y faces go from row to row by shuffle and from warp to warp through shared
// memory, and the cells come by cp.async some steps ahead (sweep2d_pf, and sweep2d_hi for cells of
// several moments).
#pragma once
#include <type_traits>

#include "rb_quot.cuh"
#include "rb_sweep_md.cuh"
#include "rb_tc.cuh"

#define RB_OCT_TILE 16   // tile edge in pencils (3D): 16×16 pencils, one per thread

namespace rb {

// octant batches: octant o's directions cut into ceil(count/db) batches of at most db
__device__ __forceinline__ int oct_groups(const DevProblem &P, int db) {
    int ng = 0;
    for (int o = 0; o < P.noct; o++) ng += (P.oct_start[o + 1] - P.oct_start[o] + db - 1) / db;
    return ng;
}
__device__ __forceinline__ int oct_group(const DevProblem &P, int db, int g, int &first, int &cnt) {
    for (int o = 0; o < P.noct; o++) {
        const int c = P.oct_start[o + 1] - P.oct_start[o], nb = (c + db - 1) / db;
        if (g < nb) {
            first = P.oct_start[o] + g * db;
            cnt = min(db, c - g * db);
            return o;
        }
        g -= nb;
    }
    first = 0;
    cnt = 0;
    return 0;
}

// The problem is a one-moment 2D/3D problem (every closure of order 1).
__host__ __device__ __forceinline__ bool one_moment_md(const DevProblem &P) {
    return P.nm5 == 1 && P.nmf[0] == 1 && P.nmf[1] == 1 && (P.ndims < 3 || P.nmf[2] == 1) && P.nm4 == 1;
}

// Directions a thread solves per cell at the most: by its registers (FP64: fx, fy, the cell's and
// the next cell's inputs are 20 registers each for 10 directions).
template <typename R> struct OctDB { static constexpr int value = 10; };
template <> struct OctDB<float> { static constexpr int value = 12; };

#define RB_OCT_MAXNX 1024  // x widths whose inverses the sweep keeps in shared memory
#define RB_OCT_PUB 2       // a CTA publishes its progress every RB_OCT_PUB steps (and after its last)
#define RB_OCT_PUBLISHER 128  // the thread that publishes

// Directions per octant batch: the octants are cut into as many batches as give every CTA of the
// team a task in one round (a step's time is nearly proportional to its directions, its number of
// steps is not), at least as many as the registers need, in even sizes (pair loads).
__device__ __forceinline__ int oct_db(const DevProblem &P, int ncta, int ntiles, int dbmax) {
    int cmax = 1;
    for (int o = 0; o < P.noct; o++) cmax = max(cmax, P.oct_start[o + 1] - P.oct_start[o]);
    const int need = (cmax + dbmax - 1) / dbmax, room = ncta / (ntiles * P.noct);
    const int nb = max(need, min(room, (cmax + 1) / 2));
    const int db = (cmax + nb - 1) / nb;
    return min(dbmax, db > 1 ? (db + 1) & ~1 : 1);
}

// Shared-memory plan of the 3D octant sweep (byte offsets, each array 16-byte aligned): two stages
// of the upwind faces of the tile's first row and layer of pencils and of every warp's cells
// (angular source / flux and energy-face flux), the z-face hand-off between pencils
// (double-buffered by step parity), the direction constants of the octant batch, the inverse x
// widths, the per-material cell terms, and the materials of the tile's cells (a byte each, rows
// padded so that a warp's 32 rows fall into different banks; longer pencils read them from memory).
#define RB_OCT_MATNX 96  // longest pencil whose materials are kept in shared memory
template <typename R>
struct Oct3dSmem {
    static constexpr long long DB = OctDB<R>::value, T = RB_OCT_TILE, TP = T * T;
    static constexpr long long RS = (long long)sizeof(R);
    static constexpr int DC = sizeof(R) == 8 ? 6 : 8;                        // constants per direction, padded to 16 bytes
    static constexpr long long CS = DB % 4 == 2 ? DB : DB + 2;               // widest cell stride of a stage (below)
    static constexpr int MROW = RB_OCT_MATNX + 4;                            // bytes of a pencil's materials
    static constexpr long long al(long long b) { return (b + 15) & ~15LL; }
    static constexpr long long fy = 0;                                      // double [2][T][DB]
    static constexpr long long fz = fy + al(2 * T * DB * 8);                // double [2][T][DB]
    static constexpr long long dc = fz + al(2 * T * DB * 8);                // R [DB][DC]
    static constexpr long long sfz = dc + al(DB * DC * RS);                 // R [2][DB][TP]
    static constexpr long long yo = sfz + al(2 * DB * TP * RS);             // R [2][DB][T] y faces leaving the tile
    static constexpr long long qb = yo + al(2 * DB * T * RS);               // R [2][TP][CS]
    static constexpr long long ix = qb + al(2 * CS * TP * RS);              // R [RB_OCT_MAXNX]
    static constexpr long long ms = ix + al(RB_OCT_MAXNX * RS);             // R [RB_MAXMAT]
    static constexpr long long mq = ms + al(RB_MAXMAT * RS);                // R [RB_MAXMAT]
    static constexpr long long mt = mq + al(RB_MAXMAT * RS);                // byte [TP][MROW]
    static constexpr long long eb = mt + al(TP * MROW);                     // double [2][TP][CS] (CSD)
    static constexpr long long bytes(bool csd) { return eb + (csd ? al(2 * CS * TP * 8) : 0); }
};
template <typename R>
__host__ __device__ constexpr long long oct3d_smem(bool csd) { return Oct3dSmem<R>::bytes(csd); }

// Tile height in y: a power of two up to RB_OCT_TILE, so that a pencil's lower neighbour is the
// previous lane of the same warp.
__host__ __device__ __forceinline__ int oct_ty(int ny) {
    int ty = 1;
    while (ty * 2 <= ny && ty * 2 <= RB_OCT_TILE) ty *= 2;
    return ty;
}

// The 3D octant sweep applies: one-moment cells, one octant batch's tiles fit in the team, every
// CTA of the team has a progress flag, and the step and round counts fit their bit fields.
__host__ __device__ __forceinline__ bool oct3d_ok(const DevProblem &P, int ncta, long long smem_bytes, int mixed) {
    if (P.ndims != 3 || !one_moment_md(P) || ncta > RB_OCT_MAXCTA) return false;
    if (P.nx + 2 * RB_OCT_TILE >= (1 << 20) || P.nd >= (1 << 12)) return false;
    const int TY = oct_ty(P.ny), TZ = P.nz < RB_OCT_TILE ? P.nz : RB_OCT_TILE;
    const int ntiles = ((P.ny + TY - 1) / TY) * ((P.nz + TZ - 1) / TZ);
    const long long need = mixed ? oct3d_smem<float>(P.csd) : oct3d_smem<double>(P.csd);
    return ntiles <= ncta && smem_bytes >= need;
}

// The angular arrays' offset of direction n at x column 0 (in sweep order) of pencil (qy, qz) of an
// octant's sweep (fx, fy, fz: along the axis or against it); a column further is ±nd from there.
// 64 bits: 2^32 values are 416×192×192 cells with the 288 directions of S16.
__host__ __device__ __forceinline__ long long oct_offset(const DevProblem &P, bool fx, bool fy, bool fz, int qy, int qz, int n) {
    const long long row = (fy ? qy : P.ny - 1 - qy) + (long long)P.ny * (fz ? qz : P.nz - 1 - qz);
    return P.nd * (P.nx * row + (fx ? 0 : P.nx - 1)) + n;
}

// asynchronous global -> shared copies (cp.async, L1-allocating), and their groups
template <int B>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(B)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// progress flags between the CTAs of a team (GPU-scope release / acquire)
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Waits until *f >= target; `seen` keeps the last value read. Gives up (false) after a bounded
// number of polls (about a second), so a wait can never hang the GPU.
__device__ __forceinline__ bool wait_progress(const unsigned long long *f, unsigned long long target,
                                              unsigned long long &seen) {
    if (seen >= target) return true;
    for (int it = 0; it < (1 << 24); it++) {
        seen = ld_acquire_u64(f);
        if (seen >= target) return true;
        if (it >= 32) __nanosleep(64);
    }
    return false;
}

// the six constants of a direction, as 16-byte loads
__device__ __forceinline__ void load6(double (&d)[6], const double *p) {
#pragma unroll
    for (int i = 0; i < 6; i += 2) {
        const double2 x = *reinterpret_cast<const double2 *>(p + i);
        d[i] = x.x;
        d[i + 1] = x.y;
    }
}
__device__ __forceinline__ void load6(float (&d)[6], const float *p) {
    const float4 x = *reinterpret_cast<const float4 *>(p);
    const float2 y = *reinterpret_cast<const float2 *>(p + 4);
    d[0] = x.x; d[1] = x.y; d[2] = x.z; d[3] = x.w; d[4] = y.x; d[5] = y.y;
}

template <typename T> struct Pair;
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };

// The sweep of one octant batch over one tile of pencils is a task; the tasks of a round (one per
// CTA) run concurrently, and a tile is paced by the tiles upwind of it in y and z: before it
// stages the faces of step s, thread 0 waits until the upwind tiles have published the steps that
// write them (s + TY − 1 and s + TZ − 1 of their own counts). A CTA publishes the number of steps
// it has completed, tagged with the sweep's epoch and the round, after a barrier that follows the
// face stores and a GPU-scope fence, so a downstream tile runs about TY steps behind its upwind
// tile with no team barrier inside the sweep.
//
// What bounds it: the L1 line lookups of a step (about two cycles each) and the chain barrier,
// faces, cells, barrier. A lane that reads its own cell's directions touches a line per lane and
// load, so a warp's 32 cells are staged together, cnt / VW neighbouring lanes on the run of one
// cell, with each lane's pencils and offsets worked out once per task; the same lanes write the
// results back. VW = 2: the batch's directions start and count even (pairs). Sweep at 64³, S8, mixed,
// mean of a solve's passes: 2070 us (element-wise staging, addresses per element), 1030 (staged by warps),
// 810 now (faces leaving coalesced, |Ω|/Δ per pencil; FP32 passes 670, FP64 ones 1310).
// RECIP: the cell as sweep_3d_tiles solves it (DevProblem::recip).
template <typename R, int DB, int VW, bool CSD, bool RECIP, class Team>
__device__ __noinline__ void sweep3d_oct(Team &t, const DevProblem &P, GroupShared &gs, void *smem,
                                         const double *phiE_in, double *phiE_out, R *psi, int db) {
    using L = Oct3dSmem<R>;
    constexpr int TT = RB_OCT_TILE, TP = TT * TT, DC = L::DC, LDB = OctDB<R>::value;
    constexpr int CS = DB % 4 == 2 ? DB : DB + 2;  // cell stride of a stage: pair loads of a warp free of bank conflicts
    const int nd = P.nd, nx = P.nx, ny = P.ny, nz = P.nz, nfm = P.nfmax;
    const int TY = oct_ty(ny), TZ = min(nz, RB_OCT_TILE);
    const int nty = (ny + TY - 1) / TY, ntz = (nz + TZ - 1) / TZ, ntiles = nty * ntz;
    const int ngrp = oct_groups(P, db);
    const int gpr = (int)t.ncta / ntiles;  // octant batches per round (≥ 1: oct3d_ok)
    const int nround = (ngrp + gpr - 1) / gpr;
    const int nsteps = nx + TY + TZ - 2;
    // per-direction scratch (md_scratch_stride): exits x [ny·nz], y [nx·nz], z [nx·ny], the
    // z-face plane [nx·ny] and the y-face plane [nx·nz] handed between tiles, then the incoming
    // boundary fluxes (boundary_in_phase)
    const long long sstride = md_scratch_stride(P);
    const long long eyo = (long long)ny * nz * nfm, ezo = eyo + (long long)nx * nz * nfm;
    const long long zoff = ezo + (long long)nx * ny * nfm, yoff = zoff + (long long)nx * ny * nfm;
    const long long xin = md_in_offset(P, 0), yin = md_in_offset(P, 1), zin_ = md_in_offset(P, 2);
    unsigned char *base = reinterpret_cast<unsigned char *>(smem);
    double *fyb = reinterpret_cast<double *>(base + L::fy);
    double *fzb = reinterpret_cast<double *>(base + L::fz);
    R *dc = reinterpret_cast<R *>(base + L::dc);
    R *sfz = reinterpret_cast<R *>(base + L::sfz), *yo = reinterpret_cast<R *>(base + L::yo);
    R *idxs = reinterpret_cast<R *>(base + L::ix);
    R *mS = reinterpret_cast<R *>(base + L::ms);
    R *mQ = reinterpret_cast<R *>(base + L::mq);
    unsigned char *mt = base + L::mt;
    const int me = threadIdx.x, lane = me & 31, jy = me % TY, jz = me / TY;
    R *qb = reinterpret_cast<R *>(base + L::qb) + (me - lane) * CS;                       // this warp's [32][CS]
    double *eb = reinterpret_cast<double *>(base + L::eb) + (CSD ? (me - lane) * CS : 0);  // (stages TP·CS apart)
    const R w1x = (R)P.w1[0], w1y = (R)P.w1[1], w1z = (R)P.w1[2], w1e = (R)P.w1[3];
    const R esa = CSD ? (R)P.EsA[0] : R(0), esb = CSD ? (R)P.EsB[0] : R(0), eout = CSD ? (R)P.Eout[0] : R(0);
    // this sweep's tables: inverse x widths, and per material Σt (+ the CSD cell term) and the
    // factor of the incoming energy-face flux
    const bool xs_sm = nx <= RB_OCT_MAXNX;
    __syncthreads();
    if (xs_sm)
        for (int i = me; i < nx; i += blockDim.x) idxs[i] = (R)(1.0 / P.dx[i]);
    for (int m = me; m < P.nmat; m += blockDim.x) {
        const R sigt = (R)gs.sigt[m];
        R scs = R(0), sq = R(0);
        if (CSD) {
            scs = (R)P.scsd[m];
            sq = esa * (R)gs.sp[m] - esb * (R)gs.sm[m];
        }
        mS[m] = scs + sigt;
        mQ[m] = sq;
    }
    if (me == 0) gs.oct_epoch++;
    __syncthreads();
    const unsigned long long epoch = (unsigned long long)gs.oct_epoch;
    unsigned long long seen_y = 0, seen_z = 0;  // thread 0: the upwind flags as last read
    bool gave_up = false;
    const int *mat = P.mat;
    double *fexit = P.fexit;
    unsigned long long *flags = P.oct_flags;
    for (int rnd = 0; rnd < nround; rnd++) {
        const int g = rnd * gpr + (int)t.crank / ntiles;
        const int tile = (int)t.crank % ntiles;
        int first = 0, cnt = 0, oc = 0;
        if ((int)t.crank < gpr * ntiles && g < ngrp) oc = oct_group(P, db, g, first, cnt);
        if (cnt == 0) continue;  // uniform over the CTA
        const bool fx = !(oc & 1), fy = !(oc & 2), fz = !(oc & 4);
        const int parts = cnt / VW;
        const int tyq = tile % nty, tzq = tile / nty;  // tile coordinates in sweep order
        const int iyy = tyq * TY + jy, izz = tzq * TZ + jz;
        const bool pok = me < TY * TZ && iyy < ny && izz < nz;
        const int iy = fy ? iyy : ny - 1 - iyy, iz = fz ? izz : nz - 1 - izz;
        const unsigned long long tagr = (epoch << 32) | ((unsigned long long)rnd << 20);
        const unsigned long long *upy = tyq > 0 ? flags + (t.crank - 1) : nullptr;
        const unsigned long long *upz = tzq > 0 ? flags + (t.crank - nty) : nullptr;
        __syncthreads();  // the previous round's readers of the region are done
        if (me < LDB) {
            const int n = first + me;
            for (int a = 0; a < 3; a++) {
                const long long blk = (long long)n * 3 + a;
                const double ac = RECIP ? 1.0 : (me < cnt ? fabs(P.cosv[(long long)a * nd + n]) : 0.0);
                dc[me * DC + a] = me < cnt ? (R)(ac * P.G[blk]) : R(0);
                dc[me * DC + 3 + a] = me < cnt ? (R)(ac * P.Gsrc[blk * nfm]) : R(0);
            }
        }
        // one-moment cells: the face closure's coefficient does not depend on the direction
        const R gox = (R)P.Gout[(long long)first * 3 * nfm], goy = (R)P.Gout[((long long)first * 3 + 1) * nfm];
        const R goz = (R)P.Gout[((long long)first * 3 + 2) * nfm];
        // the last pencils of the tile, whose faces leave it
        const int jyE = min(TY, ny - tyq * TY) - 1, jzE = min(TZ, nz - tzq * TZ) - 1;
        // The faces entering the tile in a step, one direction of one pencil per item: pencils
        // (0, j) for y faces, then (j, 0) for z faces; a thread has up to NI of them.
        constexpr int NI = (2 * TT * DB + TP - 1) / TP;
        const double *isrc[NI];  // the item's face at x column 0
        double *iout[NI];        // and the same item's face leaving the tile, from its last pencils
        int ij[NI], idst[NI];    // its pencil's offset in steps (−1: none) and place in a stage
        int io[NI], iv[NI];      // the leaving face's offset in steps and place in yo (≥ 0) or sfz (−1 − place)
        {
            const int nfy = TZ * cnt, nfz = TY * cnt;
#pragma unroll
            for (int u = 0; u < NI; u++) {
                const int e = me + u * TP;
                ij[u] = -1;
                isrc[u] = nullptr;
                iout[u] = nullptr;
                io[u] = iv[u] = 0;
                idst[u] = 0;
                if (e < nfy + nfz) {
                    const bool isy = e < nfy;
                    const int e2 = isy ? e : e - nfy, j = e2 / cnt, kk = e2 - j * cnt;
                    const int qy = tyq * TY + (isy ? 0 : j), qz = tzq * TZ + (isy ? j : 0);
                    if (qy < ny && qz < nz) {
                        const int row = isy ? (fz ? qz : nz - 1 - qz) : (fy ? qy : ny - 1 - qy);
                        const long long off = isy ? (tyq == 0 ? yin : yoff) : (tzq == 0 ? zin_ : zoff);
                        isrc[u] = fexit + (long long)(first + kk) * sstride + off + (long long)nx * row * nfm;
                        ij[u] = j;
                        const long long out = isy ? (tyq == nty - 1 ? eyo : yoff) : (tzq == ntz - 1 ? ezo : zoff);
                        iout[u] = fexit + (long long)(first + kk) * sstride + out + (long long)nx * row * nfm;
                        io[u] = j + (isy ? jyE : jzE);
                        iv[u] = isy ? kk * TT + j : -1 - (kk * TP + jzE * TY + j);
                        idst[u] = (isy ? 0 : (int)((L::fz - L::fy) / 8)) + j * LDB + kk;
                    }
                }
            }
        }
        // thread 0: the upwind tiles have published the steps that write the faces of step s
        auto wait_up = [&](int s) {
            if (me != 0 || gave_up || s >= nsteps) return;
            bool ok = true;
            if (upy) ok = wait_progress(upy, tagr | (unsigned long long)(min(s + TY - 1, nsteps - 1) + 1), seen_y);
            if (ok && upz) ok = wait_progress(upz, tagr | (unsigned long long)(min(s + TZ - 1, nsteps - 1) + 1), seen_z);
            if (!ok) {
                gave_up = true;
                atomicOr(P.status, RB_DEV_TIMEOUT);
            }
        };
        auto stage_faces = [&](int s) {
            if (s < nsteps) {
#pragma unroll
                for (int u = 0; u < NI; u++) {
                    const int ixx = s - ij[u];
                    if (ij[u] >= 0 && ixx >= 0 && ixx < nx)
                        cp_async<8>(fyb + (s & 1) * (TT * LDB) + idst[u], isrc[u] + (long long)(fx ? ixx : nx - 1 - ixx) * nfm);
                }
            }
            cp_async_commit();
        };
        // the faces that step s left to the downstream tiles (or the domain), an item per thread
        auto store_faces = [&](int s) {
            const int b = s & 1;
#pragma unroll
            for (int u = 0; u < NI; u++) {
                const int ixx = s - io[u];
                if (ij[u] >= 0 && ixx >= 0 && ixx < nx) {
                    const R f = iv[u] >= 0 ? yo[b * LDB * TT + iv[u]] : sfz[b * LDB * TP - 1 - iv[u]];
                    iout[u][(long long)(fx ? ixx : nx - 1 - ixx) * nfm] = (double)f;
                }
            }
        };
        const R idy = pok ? (R)(1.0 / P.dy[iy]) : R(0), idz = pok ? (R)(1.0 / P.dz[iz]) : R(0);
        const long long c0 = (long long)nx * (iy + ny * iz);  // the pencil's first cell
        const int dstep = jy + jz;                          // the pencil's first step
        // element e = lane + 32·i of the warp's cells: part e % parts of pencil e / parts: its offset
        // in ψ at x column −(steps it runs behind), its steps behind, its place in a stage
        constexpr int NE = DB / VW;
        long long eo[NE];
        int ed[NE], ep[NE];
        const long long estep = fx ? nd : -nd;  // a column further
#pragma unroll
        for (int i = 0; i < NE; i++) {
            const int e = lane + 32 * i, pl = e / parts, part = e - pl * parts;
            const int pm = (me - lane) + (pl < 32 ? pl : 0), py = pm % TY, pz = pm / TY;
            const int qy = tyq * TY + py, qz = tzq * TZ + pz;
            const bool ok = i < parts && pm < TY * TZ && qy < ny && qz < nz;
            ed[i] = ok ? py + pz : 1 << 28;
            ep[i] = pl * CS + part * VW;
            eo[i] = ok ? oct_offset(P, fx, fy, fz, qy, qz, first + part * VW) - ed[i] * estep : 0;
        }
        // the warp's cells of step s into stage s & 1
        auto stage_cells = [&](int s) {
            const int st = (s & 1) * (TP * CS);
#pragma unroll
            for (int i = 0; i < NE; i++) {
                if (i < parts && (unsigned)(s - ed[i]) < (unsigned)nx) {
                    const long long o = eo[i] + s * estep;
                    cp_async<VW * (int)sizeof(R)>(qb + st + ep[i], psi + o);
                    if (CSD && phiE_in) cp_async<VW * 8>(eb + st + ep[i], phiE_in + o);
                }
            }
        };
        auto store_cells = [&](int s) {
            const int st = (s & 1) * (TP * CS);
#pragma unroll
            for (int i = 0; i < NE; i++) {
                if (i < parts && (unsigned)(s - ed[i]) < (unsigned)nx) {
                    const long long o = eo[i] + s * estep;
                    if constexpr (VW == 2) {
                        using R2 = typename Pair<R>::type;
                        *reinterpret_cast<R2 *>(psi + o) = *reinterpret_cast<const R2 *>(qb + st + ep[i]);
                        if (CSD && phiE_out)
                            *reinterpret_cast<double2 *>(phiE_out + o) = *reinterpret_cast<const double2 *>(eb + st + ep[i]);
                    } else {
                        psi[o] = qb[st + ep[i]];
                        if (CSD && phiE_out) phiE_out[o] = eb[st + ep[i]];
                    }
                }
            }
        };
        const bool mat_sm = nx <= RB_OCT_MATNX;
        if (mat_sm)  // materials of the tile's pencils, a row per warp
            for (int p = me >> 5; p < TP; p += RB_THREADS / 32) {
                const int qy = tyq * TY + p % TY, qz = tzq * TZ + p / TY;
                if (p < TY * TZ && qy < ny && qz < nz) {
                    const int *m = mat + (long long)nx * ((fy ? qy : ny - 1 - qy) + ny * (fz ? qz : nz - 1 - qz));
                    for (int x = lane; x < nx; x += 32) mt[p * L::MROW + x] = (unsigned char)m[x];
                }
            }
        R fxs[DB], fyl[DB];
        {
            const long long o = xin + (iy + (long long)ny * iz) * nfm;  // the domain's incoming x faces
#pragma unroll
            for (int k = 0; k < DB; k++) {
                fyl[k] = R(0);
                fxs[k] = (pok && k < cnt) ? (R)fexit[(long long)(first + k) * sstride + o] : R(0);
            }
        }
        // RECIP: h = |Ω|/Δ per axis, the pencil's y and z ones once, the x ones where the width changes
        // (dxn: the next cell's width, loaded a step ahead; NaN: none yet). The three FP64 quotients
        // per cell and direction bounded the FP64 passes of a mixed solve: 64³, S8, two groups
        // 62.8 ms with them, 58.8 so.
        R hx[RECIP ? DB : 1], hy[RECIP ? DB : 1], hz[RECIP ? DB : 1], dxc = R(NAN), dxn = R(0);
        if constexpr (RECIP) {
            dxn = P.dx[fx ? 0 : nx - 1];
#pragma unroll
            for (int k = 0; k < DB; k++) {
                const bool in = pok && k < cnt;
                hx[k] = R(0);
                hy[k] = in ? quot(fabs(P.cosv[nd + first + k]), P.dy[iy]) : R(0);
                hz[k] = in ? quot(fabs(P.cosv[2 * nd + first + k]), P.dz[iz]) : R(0);
            }
        }
        wait_up(0);
        __syncthreads();
        stage_cells(0);
        stage_faces(0);
        for (int sg = 0; sg < nsteps; sg++) {
            wait_up(sg + 1);
            cp_async_wait<0>();  // this thread's copies of step sg have landed
            __syncthreads();     // everyone's; step sg − 1 solved; step sg + 1's faces are written
            // the faces of steps < sg − 1 are stored: publish (the barrier orders every thread's stores
            // before the release), by another warp than the one that waits for the upwind tiles
            if (me == RB_OCT_PUBLISHER && sg > 1 && (sg - 1) % RB_OCT_PUB == 0)
                st_release_u64(flags + t.crank, tagr | (unsigned long long)(sg - 1));
            if (sg > 0) store_faces(sg - 1);
            if (sg + 1 < nsteps) stage_cells(sg + 1);
            stage_faces(sg + 1);
            const int ixx = sg - dstep;
            const int rd = (sg + 1) & 1, wr = sg & 1;
            R fyi[DB];
#pragma unroll
            for (int k = 0; k < DB; k++) fyi[k] = __shfl_up_sync(0xffffffffu, fyl[k], 1);
            if (pok && ixx >= 0 && ixx < nx) {
                const int ix = fx ? ixx : nx - 1 - ixx;
                R fzi[DB];
                R *qc = qb + wr * (TP * CS) + lane * CS;
                double *ec = eb + wr * (TP * CS) + lane * CS;
                if (jy == 0) {
#pragma unroll
                    for (int k = 0; k < DB; k++) fyi[k] = (R)fyb[(wr * TT + jz) * LDB + k];
                }
                if (jz == 0) {
#pragma unroll
                    for (int k = 0; k < DB; k++) fzi[k] = (R)fzb[(wr * TT + jy) * LDB + k];
                } else {
#pragma unroll
                    for (int k = 0; k < DB; k++) fzi[k] = sfz[(rd * LDB + k) * TP + me - TY];
                }
                R v[DB], fe[CSD ? DB : 1];
                if constexpr (VW == 2) {
#pragma unroll
                    for (int k = 0; k < DB; k += 2) {
                        const auto x = *reinterpret_cast<const typename Pair<R>::type *>(qc + k);
                        v[k] = x.x;
                        v[k + 1] = x.y;
                        if constexpr (CSD) {
                            double2 e = make_double2(0.0, 0.0);
                            if (phiE_in) e = *reinterpret_cast<const double2 *>(ec + k);
                            fe[k] = (R)e.x;
                            fe[k + 1] = (R)e.y;
                        }
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < DB; k++) {
                        v[k] = qc[k];
                        if (CSD) fe[CSD ? k : 0] = phiE_in ? (R)ec[k] : R(0);
                    }
                }
                const int m = mat_sm ? mt[me * L::MROW + ix] : mat[c0 + ix];
                const R S0 = mS[m], sq = mQ[m];
                const R idx = xs_sm ? idxs[ix] : (R)(1.0 / P.dx[ix]);
                if constexpr (RECIP) {
                    if (dxn != dxc) {  // another width than the last cell's
                        dxc = dxn;
#pragma unroll
                        for (int k = 0; k < DB; k++)
                            if (k < cnt) hx[k] = quot(fabs(P.cosv[first + k]), dxc);
                    }
                    dxn = P.dx[ixx + 1 < nx ? (fx ? ix + 1 : ix - 1) : ix];
#pragma unroll
                    for (int k = 0; k < DB; k++) {
                        if (k >= cnt) continue;
                        R d[6];
                        load6(d, dc + k * DC);
                        R S = S0, q = v[k];
                        S += hx[k] * d[0];
                        S += hy[k] * d[1];
                        S += hz[k] * d[2];
                        q += hx[k] * (d[3] * fxs[k]);
                        q += hy[k] * (d[4] * fyi[k]);
                        q += hz[k] * (d[5] * fzi[k]);
                        v[k] = q * quot(1.0, S);
                        fxs[k] = w1x * fxs[k] + gox * v[k];
                        fyi[k] = w1y * fyi[k] + goy * v[k];
                        fzi[k] = w1z * fzi[k] + goz * v[k];
                    }
                } else {
                    // every direction's collision term and right-hand side, then the quotients, then the
                    // faces: three loops without a branch, so that the directions' chains overlap.
                    // FP32 takes the approximate division, whose 2-ulp error the FP64 defect correction absorbs.
                    R S[DB];
                    bool fast = true;
#pragma unroll
                    for (int k = 0; k < DB; k++) {
                        R d[6];
                        load6(d, dc + k * DC);
                        S[k] = S0 + d[0] * idx + d[1] * idy + d[2] * idz;
                        R q = v[k] + (d[3] * idx) * fxs[k] + (d[4] * idy) * fyi[k] + (d[5] * idz) * fzi[k];
                        if (CSD) q -= sq * fe[CSD ? k : 0];
                        v[k] = q;
                        if constexpr (sizeof(R) == 8) fast &= (k >= cnt) | (quot_in(q) & quot_div_in(S[k]));
                    }
                    if (fast) {
#pragma unroll
                        for (int k = 0; k < DB; k++) {
                            if constexpr (sizeof(R) == 8) v[k] = quot_by(v[k], S[k], quot_rcp(S[k]));
                            else v[k] = __fdividef(v[k], S[k]);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < DB; k++) v[k] = v[k] / S[k];
                    }
#pragma unroll
                    for (int k = 0; k < DB; k++) {
                        fxs[k] = w1x * fxs[k] + gox * v[k];
                        fyi[k] = w1y * fyi[k] + goy * v[k];
                        fzi[k] = w1z * fzi[k] + goz * v[k];
                    }
                }
#pragma unroll
                for (int k = 0; k < DB; k++)
                    if (k < cnt) sfz[(wr * LDB + k) * TP + me] = fzi[k];
                if constexpr (VW == 2) {
#pragma unroll
                    for (int k = 0; k < DB; k += 2) {
                        typename Pair<R>::type x;
                        x.x = v[k];
                        x.y = v[k + 1];
                        *reinterpret_cast<typename Pair<R>::type *>(qc + k) = x;
                        if (CSD && phiE_out)
                            *reinterpret_cast<double2 *>(ec + k) =
                                make_double2((double)(w1e * fe[CSD ? k : 0] + eout * v[k]), (double)(w1e * fe[CSD ? k + 1 : 0] + eout * v[k + 1]));
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < DB; k++) {
                        qc[k] = v[k];
                        if (CSD) ec[k] = (double)(w1e * fe[CSD ? k : 0] + eout * v[k]);
                    }
                }
                if (jy == jyE) {  // (the z faces are in sfz)
#pragma unroll
                    for (int k = 0; k < DB; k++)
                        if (k < cnt) yo[(wr * LDB + k) * TT + jz] = fyi[k];
                }
            }
#pragma unroll
            for (int k = 0; k < DB; k++) fyl[k] = fyi[k];
            __syncwarp();
            store_cells(sg);
            __syncwarp();  // before the stage takes the step after the next
        }
        cp_async_wait<0>();
        __syncthreads();
        store_faces(nsteps - 1);
        if (pok) {  // the x faces leaving the domain
            double *f = fexit + (long long)first * sstride + (iy + (long long)ny * iz) * nfm;
#pragma unroll
            for (int k = 0; k < DB; k++)
                if (k < cnt) f[(long long)k * sstride] = (double)fxs[k];
        }
        __syncthreads();
        if (me == RB_OCT_PUBLISHER) st_release_u64(flags + t.crank, tagr | (unsigned long long)nsteps);
    }
    __syncthreads();
}

// the octant sweep with the smallest instantiated batch that holds the problem's
template <typename R, bool CSD, class Team>
__device__ __forceinline__ void sweep3d_run(Team &t, const DevProblem &P, GroupShared &gs, void *smem,
                                            const double *phiE_in, double *phiE_out, R *psi) {
    const int TY = oct_ty(P.ny), TZ = min(P.nz, RB_OCT_TILE);
    const int db = oct_db(P, (int)t.ncta, ((P.ny + TY - 1) / TY) * ((P.nz + TZ - 1) / TZ), OctDB<R>::value);
    // pairs: every octant starts even and has an even count, and so do its batches
    bool even = P.nd % 2 == 0 && db % 2 == 0;
    for (int o = 0; o < P.noct; o++) even = even && (P.oct_start[o + 1] - P.oct_start[o]) % 2 == 0;
#define RB_OCT_RUN(DB_)                                                                                     \
    {                                                                                                       \
        if (even) sweep3d_oct<R, DB_, 2, CSD, false>(t, P, gs, smem, phiE_in, phiE_out, psi, db);           \
        else sweep3d_oct<R, DB_, 1, CSD, false>(t, P, gs, smem, phiE_in, phiE_out, psi, db);                \
        return;                                                                                             \
    }
    if constexpr (std::is_same<Team, GridTeam>::value) {
        if constexpr (sizeof(R) == 8 && !CSD) {
            if (P.recip) {  // (one instantiation each: three of a group's passes)
                if (even) sweep3d_oct<R, 10, 2, false, true>(t, P, gs, smem, phiE_in, phiE_out, psi, db);
                else sweep3d_oct<R, 10, 1, false, true>(t, P, gs, smem, phiE_in, phiE_out, psi, db);
                return;
            }
        }
        if (db <= 6) RB_OCT_RUN(6)
        if (sizeof(R) == 4 && db <= 10) RB_OCT_RUN(10)
    }
    RB_OCT_RUN(OctDB<R>::value)
#undef RB_OCT_RUN
}

// 2D, one-moment cells: sweep_md's wavefront with the arithmetic in R (FP64 or FP32) over an
// angular buffer held cells fastest.
//
// A warp takes 32 rows of a direction, one per lane, each a column behind the lane below; the y
// face goes up by shuffle. Lane 31 leaves its faces in shared memory for lane 0 of the warp above,
// which runs RB_2D_K more steps behind than it must, so that one block barrier per piece of RB_2D_K
// steps stands between the faces' stores and their loads.
//
// What bounds it: with one or two directions a CTA there is about one warp per scheduler, so every
// instruction of a step counts with its latency, nx + rows + lag times. So a piece of RB_2D_K steps
// works out its cells' coefficients (collision term, reciprocal, face factors: independent of the
// faces) together, in registers, and a step is left with the shuffle and the cell's few dependent
// operations. The piece's inputs come by cp.async two pieces ahead into the warp's own tile, 8 lanes
// to a row's run of 8 cells; the outputs leave the same way. 128×128, S12, FP64: 250 us (one load per
// cell in flight, a barrier per step), 130 (8 loads ahead), 95 now.
#define RB_2D_K 8
// elements of a warp's tile of one array: 32 rows of K cells, padded to an odd stride
#define RB_2D_TILE (32 * (RB_2D_K + 1))
// bytes of the sweep's region: two tiles per warp of ψ, energy-face flux and material, then Σt (+ the
// CSD cell term) and the factor of the incoming energy-face flux per material, and the inverse widths
__host__ __device__ __forceinline__ long long sweep2d_bytes(int nx, int mixed, int csd) {
    return (long long)(RB_THREADS / 32) * 2 * RB_2D_TILE * ((mixed ? 4 : 8) + (csd ? 8 : 0) + 4) + (long long)(nx + 2 * RB_MAXMAT) * (mixed ? 4 : 8);
}
template <typename R, bool CSD, class Team>
__device__ __noinline__ void sweep2d_pf(Team &t, const DevProblem &P, GroupShared &gs, void *region, const double *phiE_in,
                                        double *phiE_out, R *psi) {
    constexpr int K = RB_2D_K, TS = RB_2D_TILE, NW = RB_THREADS / 32;
    static_assert(K == 8, "a piece is 8 cells of a row: 8 lanes, 4 rows per copy");
    const int nd = P.nd, nx = P.nx, ny = P.ny, nfm = P.nfmax, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ncta = (int)t.ncta, crank = (int)t.crank;
    const int dlo = (int)((long long)nd * crank / ncta), dhi = (int)((long long)nd * (crank + 1) / ncta);
    const int my_dirs = dhi - dlo;
    if (my_dirs == 0) return;
    const int nwd = min(NW, (ny + 31) / 32), rows = 32 * nwd;  // warps of a direction, rows of a block
    int D = NW / nwd;                                          // directions in work
    const int dmax = RB_TILE_DOUBLES * (int)(sizeof(double) / sizeof(R)) / nx;  // y-face slots
    if (D > dmax) D = dmax;
    const int nrb = (ny + rows - 1) / rows;
    const int npiece = (nx + 31 + (nwd - 1) * (32 + K) + K - 1) / K;
    const long long sstride = md_scratch_stride(P), sn = P.psi_sn;
    const long long xin = md_in_offset(P, 0), yin = md_in_offset(P, 1);
    R *yface = reinterpret_cast<R *>(gs.tile);  // [D][nx]
    const R w1x = (R)P.w1[0], w1y = (R)P.w1[1], w1e = (R)P.w1[3];
    const R esa = CSD ? (R)P.EsA[0] : R(0), esb = CSD ? (R)P.EsB[0] : R(0), eout = CSD ? (R)P.Eout[0] : R(0);
    const int *mat = P.mat;
    const double *dxp = P.dx;
    // this warp's tiles [2][TS], and the inverse widths
    double *es = reinterpret_cast<double *>(region) + warp * 2 * TS;
    R *qs0 = reinterpret_cast<R *>(reinterpret_cast<double *>(region) + (CSD ? NW * 2 * TS : 0)), *qs = qs0 + warp * 2 * TS;
    int *ms0 = reinterpret_cast<int *>(qs0 + NW * 2 * TS), *ms = ms0 + warp * 2 * TS;
    R *mS = reinterpret_cast<R *>(ms0 + NW * 2 * TS), *mQ = mS + RB_MAXMAT, *idxs = mQ + RB_MAXMAT;
    __syncthreads();
    for (int m = tid; m < P.nmat; m += blockDim.x) {
        R S = (R)gs.sigt[m], sq = R(0);
        if (CSD) {
            S = (R)P.scsd[m] + S;
            sq = esa * (R)gs.sp[m] - esb * (R)gs.sm[m];
        }
        mS[m] = S;
        mQ[m] = sq;
    }
    for (int i = tid; i < nx; i += blockDim.x) idxs[i] = (R)(1.0 / dxp[i]);
    const int dl = warp / nwd, jw = warp % nwd;  // this warp's direction and its place among its warps
    const int lag0 = jw * (32 + K);              // steps the warp's first row runs behind
    for (int k0 = 0; k0 < my_dirs; k0 += D) {
        const bool active = dl < D && k0 + dl < my_dirs;
        const int n = dlo + k0 + (active ? dl : 0);
        const double mu = P.cosv[n], eta = P.cosv[nd + n];
        const bool fx = mu >= 0.0, fy = eta >= 0.0;
        const R gx = (R)(fabs(mu) * P.G[(long long)n * 3]), gy = (R)(fabs(eta) * P.G[(long long)n * 3 + 1]);
        const R sx = (R)(fabs(mu) * P.Gsrc[((long long)n * 3) * nfm]), sy = (R)(fabs(eta) * P.Gsrc[((long long)n * 3 + 1) * nfm]);
        const R ox = (R)P.Gout[((long long)n * 3) * nfm], oy = (R)P.Gout[((long long)n * 3 + 1) * nfm];
        double *scr = P.fexit + (long long)n * sstride;
        double *exx = scr, *exy = exx + (long long)ny * nfm;
        R *yf = yface + (long long)(active ? dl : 0) * nx;
        R *pn = psi + n * sn;
        const double *ein = (CSD && phiE_in) ? phiE_in + n * sn : nullptr;
        double *eou = (CSD && phiE_out) ? phiE_out + n * sn : nullptr;
        __syncthreads();  // the previous round's readers of the face slots are done
        if (active)       // the first row's Y faces: the incoming fluxes of boundary_in_phase
            for (int i = 32 * jw + lane; i < nx; i += rows) yf[i] = (R)scr[yin + (long long)(fx ? i : nx - 1 - i) * nfm];
        for (int rb = 0; rb < nrb; rb++) {
            const int iy0 = rb * rows + 32 * jw, iyy = iy0 + lane;  // the warp's first row, this row
            const bool row = active && iyy < ny;
            const int iy = fy ? iyy : ny - 1 - iyy;
            const R idy = row ? (R)(1.0 / P.dy[iy]) : R(0);
            const bool last = iyy == ny - 1, keep = lane == 31 || last;  // rows whose faces go on
            // Element i of this lane in a piece: row 4·i + lane/8, step lane%8. Its column in sweep
            // order is (first step of the piece) + eb − 4·i, its cell e0 + i·de + (first step)·dx1.
            const int er = lane >> 3, ec = lane & 7;
            const int eb = ec - lag0 - er, rmax = active ? ny - iy0 - er : 0;  // rows: 4·i < rmax
            const int dx1 = fx ? 1 : -1;
            const long long e0 = (long long)nx * (fy ? iy0 + er : ny - 1 - iy0 - er) + (fx ? eb : nx - 1 - eb);
            const long long de = 4LL * (fy ? nx : -nx) - 4LL * dx1;
            const int eo = er * (K + 1) + ec;
            auto load = [&](int p) {  // the inputs of piece p
                const int b = (p & 1) * TS + eo, c0 = p * K + eb;
                const long long g = e0 + (long long)(p * K) * dx1;
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (4 * i < rmax && (unsigned)(c0 - 4 * i) < (unsigned)nx) {
                        const long long c = g + i * de;
                        cp_async<sizeof(R)>(qs + b + i * 4 * (K + 1), pn + c);
                        if (CSD && ein) cp_async<8>(es + b + i * 4 * (K + 1), ein + c);
                        cp_async<4>(ms + b + i * 4 * (K + 1), mat + c);
                    }
                cp_async_commit();
            };
            auto store = [&](int p) {  // the outputs of piece p
                const int b = (p & 1) * TS + eo, c0 = p * K + eb;
                const long long g = e0 + (long long)(p * K) * dx1;
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (4 * i < rmax && (unsigned)(c0 - 4 * i) < (unsigned)nx) {
                        const long long c = g + i * de;
                        pn[c] = qs[b + i * 4 * (K + 1)];
                        if (CSD && eou) eou[c] = es[b + i * 4 * (K + 1)];
                    }
            };
            load(0);
            load(1);
            R F0 = row ? (R)scr[xin + (long long)iy * nfm] : R(0), Fy = R(0);
            const R cay = sy * idy;
            for (int p = 0; p < npiece; p++) {
                cp_async_wait<1>();
                __syncthreads();  // the piece in every lane's view; the faces that lane 0 takes are stored
                const int c0 = p * K - lag0 - lane;  // this row's column at the piece's first step
                R *q = qs + (p & 1) * TS + lane * (K + 1);
                double *e = es + (p & 1) * TS + lane * (K + 1);
                const int *mm = ms + (p & 1) * TS + lane * (K + 1);
                R cS[K], cr[K], cq[K], cax[K], cf[K], ce[CSD ? K : 1], cQ[CSD ? K : 1];
                bool in[K], far = false;
#pragma unroll
                for (int u = 0; u < K; u++) {
                    in[u] = row && (unsigned)(c0 + u) < (unsigned)nx;
                    const int x = in[u] ? c0 + u : 0, m = in[u] ? mm[u] : 0;
                    const R ix = idxs[fx ? x : nx - 1 - x];
                    R S = mS[m];
                    S = S + gx * ix + gy * idy;
                    cS[u] = S;
                    cq[u] = q[u];
                    cax[u] = sx * ix;
                    cf[u] = lane == 0 ? yf[x] : R(0);
                    if (CSD) {
                        ce[CSD ? u : 0] = ein ? (R)e[u] : R(0);
                        cQ[CSD ? u : 0] = mQ[m];
                    }
                }
#pragma unroll
                for (int u = 0; u < K; u++) {
                    cr[u] = quot_rcp(cS[u]);
                    far |= in[u] & !quot_div_in(cS[u]);
                }
                // X face of the row and Y face of the column (sn_sweep_2D.jl:71-132); true where a dividend
                // of the piece is outside quot_by's range
                auto steps = [&](auto divide) {
                    bool out = false;
#pragma unroll
                    for (int u = 0; u < K; u++) {
                        const R up = __shfl_up_sync(0xffffffffu, Fy, 1);
                        const R F1 = lane == 0 ? cf[u] : up;
                        R qq = cq[u] + cax[u] * F0 + cay * F1;
                        if (CSD) qq = fma(-cQ[CSD ? u : 0], ce[CSD ? u : 0], qq);
                        R v;
                        if constexpr (decltype(divide)::value) {
                            v = qq / cS[u];
                        } else {
                            v = quot_by(qq, cS[u], cr[u]);
                            out |= in[u] & !quot_in(qq);
                        }
                        const R F0o = w1x * F0 + ox * v;
                        Fy = w1y * F1 + oy * v;
                        F0 = in[u] ? F0o : F0;
                        q[u] = v;
                        if (CSD && eou) e[u] = (double)fma(w1e, ce[CSD ? u : 0], eout * v);
                        if (keep && in[u]) yf[c0 + u] = Fy;
                    }
                    return out;
                };
                const R F0p = F0, Fyp = Fy;
                far |= steps(std::false_type{});
                if (__any_sync(0xffffffffu, far)) {  // the piece again, by divisions
                    F0 = F0p;
                    Fy = Fyp;
                    steps(std::true_type{});
                }
                __syncwarp();
                store(p);
                __syncwarp();  // the tile takes the piece after the next
                load(p + 2);
            }
            if (row) exx[(long long)iy * nfm] = (double)F0;
            cp_async_wait<0>();
            __syncthreads();
            if (active && rb == nrb - 1)  // the last row's faces leave the domain
                for (int i = 32 * jw + lane; i < nx; i += rows) exy[(long long)(fx ? i : nx - 1 - i) * nfm] = (double)yf[i];
        }
    }
}

// 2D cells of NM moments (FP64): the same wavefront. The cell matrix S = Σt·I + Σ_a h_a·G_a + Scsd
// of flux_2D_BTE / flux_2D_BFP (sn_2D_bte.jl:35-116, sn_2D_bfp.jl:45-154) depends on the direction,
// the material and the widths only, so a lane keeps its inverse in registers along the row and
// factors again where the material or a width changes; a cell is then a product with the inverse.
// (The run-time shaped solve, which stays for the other shapes, eliminates every cell's matrix in
// local memory: 9.4 us a step at 41×30, S6, four moments; 0.9 here.)
#define RB_2DHI_PF 4
template <int NM, int NF, int NE, bool CSD>
struct Sweep2dHi {
    // doubles of the direction tables: G, Gsrc, Gout of both axes, the energy-face factors
    static constexpr int TAB = 2 * (NM * NM + 2 * NM * NF) + (CSD ? 3 * NM * NE : 0);
    static constexpr int SLOT = NM + (CSD ? NE : 0);
    static constexpr long long bytes = 8LL * (8 * TAB + (long long)RB_2DHI_PF * SLOT * RB_THREADS) + 4LL * RB_2DHI_PF * RB_THREADS;
    // a thread's slot is NM consecutive values, copied and stored in pairs where NM is even
    static constexpr int V = NM % 2 == 0 ? 2 : 1, VE = NE % 2 == 0 ? 2 : 1;
};
template <int NM, int NF, int NE, bool CSD, class Team>
__device__ __noinline__ void sweep2d_hi(Team &t, const DevProblem &P, GroupShared &gs, void *region, const double *phiE_in,
                                        double *phiE_out) {
    using L = Sweep2dHi<NM, NF, NE, CSD>;
    constexpr int PF = RB_2DHI_PF, K = RB_2D_K, GG = NM * NM, GF = NM * NF;
    const int nd = P.nd, nx = P.nx, ny = P.ny, nfm = P.nfmax, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ncta = (int)t.ncta, crank = (int)t.crank;
    const int dlo = (int)((long long)nd * crank / ncta), dhi = (int)((long long)nd * (crank + 1) / ncta);
    const int my_dirs = dhi - dlo;
    if (my_dirs == 0) return;
    const int nwarp = RB_THREADS / 32;
    const int nwd = min(nwarp, (ny + 31) / 32), rows = 32 * nwd;
    int D = nwarp / nwd;
    const int dmax = RB_TILE_DOUBLES / (nx * NF);  // y-face slots (at least one: checked at upload)
    if (D > dmax) D = dmax;
    const int nrb = (ny + rows - 1) / rows;
    const int nsteps = nx + 31 + (nwd - 1) * (32 + K);
    const long long sstride = md_scratch_stride(P);
    const long long xin = md_in_offset(P, 0), yin = md_in_offset(P, 1);
    double *yface = gs.tile;  // [D][nx][NF]
    double *tabs = reinterpret_cast<double *>(region);
    double *qs = tabs + 8 * L::TAB + tid * L::V;        // [PF][NM / V][threads][V]
    double *es = tabs + 8 * L::TAB + PF * NM * RB_THREADS + tid * L::VE;  // [PF][NE / VE][threads][VE]
    int *ms = reinterpret_cast<int *>(tabs + 8 * L::TAB + PF * L::SLOT * RB_THREADS) + tid;  // [PF][threads]
    double *dxs = reinterpret_cast<double *>(ms - tid + PF * RB_THREADS);  // [nx] widths
    auto qat = [](int o, int j) { return ((o * (NM / L::V) + j / L::V) * RB_THREADS) * L::V + j % L::V; };
    auto eat = [](int o, int e) { return ((o * (NE / L::VE) + e / L::VE) * RB_THREADS) * L::VE + e % L::VE; };
    for (int i = tid; i < nx; i += blockDim.x) dxs[i] = P.dx[i];
    const double w1x = P.w1[0], w1y = P.w1[1], w1e = P.w1[3];
    const int *mat = P.mat;
    const int dl = warp / nwd, jw = warp % nwd;
    const int lag = jw * (32 + K) + lane;
    for (int k0 = 0; k0 < my_dirs; k0 += D) {
        const bool active = dl < D && k0 + dl < my_dirs;
        const int n = dlo + k0 + (active ? dl : 0);
        const double amu = fabs(P.cosv[n]), aeta = fabs(P.cosv[nd + n]);
        const bool fx = P.cosv[n] >= 0.0, fy = P.cosv[nd + n] >= 0.0;
        double *scr = P.fexit + (long long)n * sstride;
        double *exx = scr, *exy = exx + (long long)ny * nfm;
        double *yf = yface + (long long)(active ? dl : 0) * nx * NF;
        double *T = tabs + (active ? dl : 0) * L::TAB;  // [a]: G, Gsrc (j + NM·f), Gout (f + NF·j); then EsA, EsB, Eout
        __syncthreads();  // the previous round's readers are done
        if (active) {
            for (int e = 32 * jw + lane; e < L::TAB; e += rows) {
                constexpr int AX = GG + 2 * GF;
                double v;
                if (e < 2 * AX) {
                    const int a = e / AX, o = e % AX;
                    const long long blk = (long long)n * 3 + a;
                    v = o < GG ? P.G[blk * GG + o] : (o < GG + GF ? P.Gsrc[blk * NM * nfm + o - GG] : P.Gout[blk * NM * nfm + o - GG - GF]);
                } else {
                    const int o = e - 2 * AX;
                    v = o < NM * NE ? P.EsA[o] : (o < 2 * NM * NE ? P.EsB[o - NM * NE] : P.Eout[o - 2 * NM * NE]);
                }
                T[e] = v;
            }
            for (int i = 32 * jw + lane; i < nx; i += rows)
                for (int f = 0; f < NF; f++) yf[i * NF + f] = scr[yin + (long long)(fx ? i : nx - 1 - i) * nfm + f];
        }
        __syncthreads();
        const double *Tx = T, *Ty = T + GG + 2 * GF, *TE = T + 2 * (GG + 2 * GF);
        for (int rb = 0; rb < nrb; rb++) {
            const int iyy = rb * rows + 32 * jw + lane;
            const bool row = active && iyy < ny;
            const int iy = fy ? iyy : ny - 1 - iyy;
            const double hy = row ? aeta / P.dy[iy] : 0.0;
            const long long c0 = row ? (long long)nx * iy : 0;
            double *prow = P.psi + n * P.psi_sn + NM * c0;
            const double *ein = (CSD && phiE_in) ? phiE_in + n * P.pe_sn + NE * c0 : nullptr;
            double *eou = (CSD && phiE_out) ? phiE_out + n * P.pe_sn + NE * c0 : nullptr;
            const bool last = iyy == ny - 1, top = lane == 31 && !last;
            auto load = [&](int s) {
                const int ixx = s - lag, o = s % PF;
                if (row && ixx >= 0 && ixx < nx) {
                    const int ix = fx ? ixx : nx - 1 - ixx;
#pragma unroll
                    for (int j = 0; j < NM; j += L::V) cp_async<8 * L::V>(qs + qat(o, j), prow + ix * NM + j);
                    if (CSD && ein)
#pragma unroll
                        for (int e = 0; e < NE; e += L::VE) cp_async<8 * L::VE>(es + eat(o, e), ein + ix * NE + e);
                    cp_async<4>(ms + o * RB_THREADS, mat + c0 + ix);
                }
                cp_async_commit();
            };
            // the direction's face factors stay in registers along the row
            double gsx[GF], gsy[GF], gox[GF], goy[GF];
#pragma unroll
            for (int e = 0; e < GF; e++) {
                gsx[e] = Tx[GG + e];
                gsy[e] = hy * Ty[GG + e];
                gox[e] = Tx[GG + GF + e];
                goy[e] = Ty[GG + GF + e];
            }
            double Si[NM * NM], F0[NF], Fy[NF], hk = -1.0, hx = 0.0, esa[CSD ? NM * NE : 1];
            int mk = -1;
#pragma unroll
            for (int e = 0; e < NM * NM; e++) Si[e] = 0.0;
#pragma unroll
            for (int f = 0; f < NF; f++) {
                F0[f] = row ? scr[xin + (long long)iy * nfm + f] : 0.0;
                Fy[f] = 0.0;
            }
            for (int s = 0; s < PF; s++) load(s);
            for (int s = 0; s < nsteps; s++) {
                const int ixx = s - lag, o = s % PF;
                const bool in = row && ixx >= 0 && ixx < nx;
                if (s % K == 0) __syncthreads();  // the faces that lane 0 loads in these steps are stored
                cp_async_wait<PF - 1>();
                double F1[NF];
#pragma unroll
                for (int f = 0; f < NF; f++) F1[f] = __shfl_up_sync(0xffffffffu, Fy[f], 1);
                if (in) {
                    const int ix = fx ? ixx : nx - 1 - ixx;
                    const int m = ms[o * RB_THREADS];
                    const double dxc = dxs[ix];
                    if (m != mk || dxc != hk) {  // another kind of cell: its inverse
                        mk = m;
                        hk = dxc;
                        hx = amu / dxc;
                        double S[NM * NM], q[NM][NM];
#pragma unroll
                        for (int i = 0; i < NM; i++)
#pragma unroll
                            for (int j = 0; j < NM; j++) {
                                S[i + NM * j] = (CSD ? P.scsd[(long long)m * GG + i + NM * j] : 0.0) + (i == j ? gs.sigt[m] : 0.0) +
                                                hx * Tx[i + NM * j] + hy * Ty[i + NM * j];
                                q[i][j] = i == j ? 1.0 : 0.0;
                            }
                        lu_solve<double, NM, NM>(S, q);
#pragma unroll
                        for (int j = 0; j < NM; j++)
#pragma unroll
                            for (int i = 0; i < NM; i++) Si[i + NM * j] = q[j][i];
                        if (CSD)
#pragma unroll
                            for (int e = 0; e < NM * NE; e++) esa[CSD ? e : 0] = TE[e] * gs.sp[m] - TE[NM * NE + e] * gs.sm[m];
                    }
                    if (lane == 0)
#pragma unroll
                        for (int f = 0; f < NF; f++) F1[f] = yf[ixx * NF + f];
                    double q[NM], v[NM], fe[CSD ? NE : 1];
#pragma unroll
                    for (int j = 0; j < NM; j++) {
                        double ax = 0.0, ay = 0.0;
#pragma unroll
                        for (int f = 0; f < NF; f++) {
                            ax += gsx[j + NM * f] * F0[f];
                            ay += gsy[j + NM * f] * F1[f];
                        }
                        q[j] = qs[qat(o, j)] + hx * ax + ay;
                    }
                    if constexpr (CSD) {
#pragma unroll
                        for (int e = 0; e < NE; e++) fe[e] = ein ? es[eat(o, e)] : 0.0;
#pragma unroll
                        for (int j = 0; j < NM; j++)
#pragma unroll
                            for (int e = 0; e < NE; e++) q[j] -= esa[j + NM * e] * fe[e];
                    }
#pragma unroll
                    for (int i = 0; i < NM; i++) {
                        double x = 0.0;
#pragma unroll
                        for (int j = 0; j < NM; j++) x += Si[i + NM * j] * q[j];
                        v[i] = x;
                    }
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        double x = w1x * F0[f], y = w1y * F1[f];
#pragma unroll
                        for (int j = 0; j < NM; j++) {
                            x += gox[f + NF * j] * v[j];
                            y += goy[f + NF * j] * v[j];
                        }
                        F0[f] = x;
                        Fy[f] = y;
                    }
#pragma unroll
                    for (int j = 0; j < NM; j += L::V) {
                        if (L::V == 2) *reinterpret_cast<double2 *>(prow + ix * NM + j) = make_double2(v[j], v[j + L::V - 1]);
                        else prow[ix * NM + j] = v[j];
                    }
                    if constexpr (CSD) {
                        if (eou)
#pragma unroll
                            for (int e = 0; e < NE; e++) {
                                double x = w1e * fe[e];
#pragma unroll
                                for (int j = 0; j < NM; j++) x += TE[2 * NM * NE + e + NE * j] * v[j];
                                eou[ix * NE + e] = x;
                            }
                    }
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        if (top) yf[ixx * NF + f] = Fy[f];
                        if (ixx == nx - 1) exx[(long long)iy * nfm + f] = F0[f];
                        if (last) exy[(long long)ix * nfm + f] = Fy[f];
                    }
                }
                __syncwarp();
                load(s + PF);
            }
            cp_async_wait<0>();
            __syncthreads();
        }
    }
}

// 2D cells of several moments: the compiled shapes (linear closures: full coupling, without and with
// an energy closure of order 1, and without cross terms), false where the shape is another one.
// sweep2d_hi_bytes is the region they need.
__host__ __device__ __forceinline__ int sweep2d_hi_shape(const DevProblem &P) {
    if (P.ndims != 2 || P.nmf[0] != P.nmf[1] || P.nfmax != P.nmf[0]) return 0;
    if (!P.csd && P.nm5 == 4 && P.nmf[0] == 2) return 1;
    if (!P.csd && P.nm5 == 3 && P.nmf[0] == 2) return 2;
    if (P.csd && P.nm5 == 4 && P.nmf[0] == 2 && P.nm4 == 4) return 3;
    return 0;
}
__host__ __device__ __forceinline__ long long sweep2d_hi_bytes(const DevProblem &P) {
    const int k = sweep2d_hi_shape(P);
    const long long fixed = k == 1 ? Sweep2dHi<4, 2, 1, false>::bytes
                                   : (k == 2 ? Sweep2dHi<3, 2, 1, false>::bytes : Sweep2dHi<4, 2, 4, true>::bytes);
    return k == 0 ? 0 : fixed + 8LL * P.nx;
}
template <class Team>
__device__ __forceinline__ bool sweep2d_hi_run(Team &t, const DevProblem &P, GroupShared &gs, void *region, long long bytes,
                                               const double *pE, double *phiE_out) {
    const int k = sweep2d_hi_shape(P);
    if (k == 0 || bytes < sweep2d_hi_bytes(P)) return false;
    if (k == 1) sweep2d_hi<4, 2, 1, false>(t, P, gs, region, pE, phiE_out);
    else if (k == 2) sweep2d_hi<3, 2, 1, false>(t, P, gs, region, pE, phiE_out);
    else sweep2d_hi<4, 2, 4, true>(t, P, gs, region, pE, phiE_out);
    return true;
}

// The pass for 2D and 3D problems. mixed: FP32 angular buffer, products and sweep where the
// cells are one-moment and (3D) the octant sweep fits the team; every other 2D/3D pass runs in
// FP64 (the result is then the plain form's).
template <class Team>
__device__ __noinline__ void pass_md(Team &t, const DevProblem &P, GroupShared &gs, void *smem, long long smem_bytes,
                        const double *zin, double *zout, int homog, int matvec, int ig, const double *phiE_in,
                        double *phiE_out, int mixed) {
    const bool one = one_moment_md(P);
    const bool oct = oct3d_ok(P, (int)t.ncta, smem_bytes, mixed);
    const bool pf = P.ndims == 2 && one && smem_bytes >= sweep2d_bytes(P.nx, 0, P.csd);
    const int mx = (mixed && (pf || oct)) ? 1 : 0;
    // the mixed form's products go to the tensor cores where the CTA holds TMEM and they fit
    if (!mx || !m2d_tc(t, P, gs, gs.tc, smem, smem_bytes, zin, homog ? nullptr : P.qnout))
        m2d_tiles(t, P, gs, smem, smem_bytes, zin, homog ? nullptr : P.qnout, P.psi, 1, mx);
    const int np_source = homog ? 0 : P.np_source;
    const double *pE = (P.csd && !homog) ? phiE_in : nullptr;
    const bool hi = sweep2d_hi_shape(P) != 0 && smem_bytes >= sweep2d_hi_bytes(P);
    const bool newsweep = (P.ndims == 3 && oct) || (P.ndims == 2 && (pf || hi));
    // the faces' products stage in the region, or in GroupShared where there is none
    const bool own = smem_bytes >= (long long)sizeof(gs.tile);
    void *fr = own ? smem : (void *)gs.tile;
    const long long frb = own ? smem_bytes : (long long)sizeof(gs.tile);
    if (newsweep) boundary_in_phase(t, P, fr, frb, zin, np_source, ig);
    t.sync();
    if (P.ndims == 3 && oct) {
        if (mx) {
            if (P.csd) sweep3d_run<float, true>(t, P, gs, smem, pE, phiE_out, P.psi32);
            else sweep3d_run<float, false>(t, P, gs, smem, pE, phiE_out, P.psi32);
        } else {
            if (P.csd) sweep3d_run<double, true>(t, P, gs, smem, pE, phiE_out, P.psi);
            else sweep3d_run<double, false>(t, P, gs, smem, pE, phiE_out, P.psi);
        }
    } else if (pf) {
        if (mx) {
            if (P.csd) sweep2d_pf<float, true>(t, P, gs, smem, pE, phiE_out, P.psi32);
            else sweep2d_pf<float, false>(t, P, gs, smem, pE, phiE_out, P.psi32);
        } else {
            if (P.csd) sweep2d_pf<double, true>(t, P, gs, smem, pE, phiE_out, P.psi);
            else sweep2d_pf<double, false>(t, P, gs, smem, pE, phiE_out, P.psi);
        }
    } else if (P.ndims == 3) {
        if (one && !P.csd) sweep_3d_tiles<CellMDfix<1, 1, 1, false, 3>, 1, 1, 1>(t, P, gs, zin, np_source, pE, phiE_out, ig);
        else if (one) sweep_3d_tiles<CellMDfix<1, 1, 1, true, 3>, 1, 1, 1>(t, P, gs, zin, np_source, pE, phiE_out, ig);
        else sweep_3d_tiles<CellMDgen, RB_MAXNM, RB_MAXFACE, RB_MAXFACE>(t, P, gs, zin, np_source, pE, phiE_out, ig);
    } else if (!hi || !sweep2d_hi_run(t, P, gs, smem, smem_bytes, pE, phiE_out)) {
        sweep_md<CellMDgen, RB_MAXNM, RB_MAXFACE, RB_MAXFACE>(t, P, gs, zin, np_source, pE, phiE_out, ig);
    }
    t.sync();
    if (!mx || !d2m_tc(t, P, gs.tc, smem, smem_bytes, zin, zout, matvec)) d2m_tiles(t, P, gs, smem, smem_bytes, zin, zout, matvec, mx);
    boundary_out_md(t, P, fr, frb, zin, zout, matvec);
    t.sync();
}

}  // namespace rb
