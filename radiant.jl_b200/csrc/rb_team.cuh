// rb_team.cuh -- the team that owns one problem: one thread-block cluster.
//
// Every phase of a transport pass and every vector operation of the in-group accelerators is
// spread over all threads of the cluster; team barriers are hardware cluster barriers.
// Reductions are deterministic and give the same bits in every thread of every CTA: each warp
// reduces by xor butterfly (commutative pairs, identical in all lanes), each CTA sums its warps
// in a fixed order and stores that partial into its own slot in every CTA of the cluster
// (distributed shared memory), and after one cluster barrier every thread adds the slots in
// rank order from its own shared memory. Slot sets alternate between two buffers, so a
// reduction costs one cluster barrier. All threads run the same control flow, which the
// identical reduction bits guarantee, so no CTA can leave a barrier sequence early.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

namespace rb {
namespace cg = cooperative_groups;

// Scratch of a reduction of up to RB_SM values (doubles): per-warp partials [8][RB_SM], per-CTA
// slots [16][RB_SM] (cluster teams), the sums [RB_SM].
#define RB_SM 96
#define RB_SM_SLOT (8 * RB_SM)
#define RB_SM_RES (RB_SM_SLOT + 16 * RB_SM)
#define RB_SM_DOUBLES (RB_SM_RES + RB_SM)
#define RB_ROW 256  // CTAs of a grid team whose partials one warp adds through shared memory

struct TeamShared {
    double part[2][16][4];  // partial sums of each CTA, double-buffered, up to 4 values per reduction
    double warp[16][4];
    int idx;            // problem index broadcast by the cluster leader
};

struct ClusterTeam {
    TeamShared *sh;
    unsigned crank;   // CTA rank in the cluster
    unsigned ncta;    // CTAs in the cluster
    int phase;        // reduction counter (selects the slot)

    __device__ void init(TeamShared *s) {
        sh = s;
        cg::cluster_group cl = cg::this_cluster();
        crank = cl.block_rank();
        ncta = cl.num_blocks();
        phase = 0;
    }
    __device__ __forceinline__ int rank() const { return (int)(crank * blockDim.x + threadIdx.x); }
    __device__ __forceinline__ int size() const { return (int)(ncta * blockDim.x); }
    __device__ __forceinline__ bool leader() const { return threadIdx.x == 0; }  // one per CTA
    __device__ __forceinline__ void sync() const { cg::this_cluster().sync(); }

    // Sum of K values over the team (K <= 4); every thread gets identical bits.
    template <int K>
    __device__ void sumk(double (&v)[K]) {
#pragma unroll
        for (int k = 0; k < K; k++)
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int k = 0; k < K; k++) sh->warp[w][k] = v[k];
        __syncthreads();
        const int slot = phase & 1;
        phase++;
        cg::cluster_group cl = cg::this_cluster();
        if (threadIdx.x < ncta) {  // thread q stores this CTA's partial into CTA q
            double s[K];
#pragma unroll
            for (int k = 0; k < K; k++) {
                s[k] = 0.0;
                for (int i = 0; i < nw; i++) s[k] += sh->warp[i][k];
            }
            double *dst = cl.map_shared_rank(&sh->part[slot][crank][0], threadIdx.x);
#pragma unroll
            for (int k = 0; k < K; k++) dst[k] = s[k];
        }
        cl.sync();
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = 0.0;
        for (unsigned r = 0; r < ncta; r++)
#pragma unroll
            for (int k = 0; k < K; k++) v[k] += sh->part[slot][r][k];
    }
    // Sums of n ≤ RB_SM values over the team at the price of one barrier: warp w left its partials
    // in scr[w·RB_SM + i] (lane 0 after a butterfly); the sums end in the returned array, the same
    // bits in every CTA. One set of slots: a team barrier (the norm's reduction, the pass) stands
    // between two calls.
    __device__ double *sum_many(double *scr, int n) {
        const int nw = (blockDim.x + 31) >> 5;
        double *slots = scr + RB_SM_SLOT, *res = scr + RB_SM_RES;
        cg::cluster_group cl = cg::this_cluster();
        __syncthreads();
        for (int e = threadIdx.x; e < n * (int)ncta; e += blockDim.x) {
            const int q = e / n, i = e - q * n;
            double s = 0.0;
            for (int w = 0; w < nw; w++) s += scr[w * RB_SM + i];
            *cl.map_shared_rank(slots + crank * RB_SM + i, q) = s;
        }
        cl.sync();
        if ((int)threadIdx.x < n) {
            double s = 0.0;
            for (unsigned r = 0; r < ncta; r++) s += slots[r * RB_SM + threadIdx.x];
            res[threadIdx.x] = s;
        }
        __syncthreads();
        return res;
    }
    __device__ double sum(double v) {
        double a[1] = {v};
        sumk<1>(a);
        return a[0];
    }
    __device__ int any(int flag) { return sum(flag ? 1.0 : 0.0) > 0.0; }
    // Index handed out by the cluster leader (CTA 0, thread 0) to the whole cluster.
    __device__ int broadcast_from_leader(int v) {
        cg::cluster_group cl = cg::this_cluster();
        if (crank == 0 && threadIdx.x == 0) sh->idx = v;
        cl.sync();
        const int r = *cl.map_shared_rank(&sh->idx, 0);
        cl.sync();
        return r;
    }
};


// A team of every CTA of a cooperative launch (one problem on the whole GPU, for 2D and 3D
// solves). Barriers are grid barriers; in a reduction every CTA writes its partial into a row of each
// CTA (double-buffered), and after the barrier one warp of every CTA adds its own row in the same
// order, so every thread of the grid sees the same bits: in CTA order for the mixed form (its FP32
// roundings follow the last bit of every Krylov scalar, so that order is part of its result), else
// lane l the CTAs l, l + 32, … and a butterfly. (One row that all 148 CTAs read after the barrier
// serialised in L2: 3 us a round of loads, and five rounds for the sum in CTA order.)
struct GridTeam {
    TeamShared *sh;
    double *gpart;    // partial sums: [2][ncta][4][ncta] of sumk, then [RB_SM][ncta] and [ncta][RB_SM] of sum_many
    unsigned crank;
    unsigned ncta;
    int phase;
    bool ordered = false;
    double *rows;     // [4][RB_ROW] shared memory free between the phases

    __device__ void init(TeamShared *s, double *gp, double *scratch) {
        sh = s;
        rows = scratch;
        gpart = gp;
        crank = blockIdx.x;
        ncta = gridDim.x;
        phase = 0;
    }
    __device__ __forceinline__ int rank() const { return (int)(crank * blockDim.x + threadIdx.x); }
    __device__ __forceinline__ int size() const { return (int)(ncta * blockDim.x); }
    __device__ __forceinline__ bool leader() const { return threadIdx.x == 0; }
    __device__ __forceinline__ void sync() const { cg::this_grid().sync(); }

    template <int K>
    __device__ void sumk(double (&v)[K]) {
#pragma unroll
        for (int k = 0; k < K; k++)
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int k = 0; k < K; k++) sh->warp[w][k] = v[k];
        __syncthreads();
        const int slot = phase & 1;
        phase++;
        double *gp = gpart + (long long)slot * 4 * ncta * ncta;  // [to][4][from]
        double ps[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
            ps[k] = 0.0;
            for (int i = 0; i < nw; i++) ps[k] += sh->warp[i][k];
        }
        for (unsigned q = threadIdx.x; q < ncta; q += blockDim.x)
#pragma unroll
            for (int k = 0; k < K; k++) gp[((long long)q * 4 + k) * ncta + crank] = ps[k];
        cg::this_grid().sync();
        if (w < K) {
            const double s = rank_sum(gp + ((long long)crank * 4 + w) * ncta, rows + w * RB_ROW);
            if ((threadIdx.x & 31) == 0) sh->part[slot][0][w] = s;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = sh->part[slot][0][k];
    }
    // Sum of one value over the CTAs, by one warp (the same bits in every lane). In CTA order: the
    // partials through `row` (shared memory of the warp, ncta doubles), read back one after another.
    __device__ __forceinline__ double rank_sum(const double *p, double *row) const {
        const unsigned n = ncta, lane = threadIdx.x & 31;
        double s = 0.0;
        if (ordered && n <= RB_ROW) {
#pragma unroll 5
            for (unsigned r = lane; r < n; r += 32) row[r] = p[r];
            __syncwarp();
#pragma unroll 8
            for (unsigned r = 0; r < n; r++) s += row[r];
            __syncwarp();
            return s;
        }
        if (ordered) {
            for (unsigned r = 0; r < n; r++) s += p[r];
            return s;
        }
#pragma unroll 8
        for (unsigned r = lane; r < n; r += 32) s += p[r];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    }
    // as ClusterTeam::sum_many: CTA i adds value i's partials and writes the sum into a row of each
    // CTA (two barriers, and no line that every CTA reads)
    __device__ double *sum_many(double *scr, int n) {
        const int nw = (blockDim.x + 31) >> 5, w = threadIdx.x >> 5;
        double *gp = gpart + 8LL * ncta * ncta, *gr = gp + (long long)RB_SM * ncta, *res = scr + RB_SM_RES;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            double s = 0.0;
            for (int q = 0; q < nw; q++) s += scr[q * RB_SM + i];
            gp[(long long)i * ncta + crank] = s;
        }
        cg::this_grid().sync();
        for (int i = (int)crank; i < n; i += (int)ncta) {
            if (w == 0) {
                const double s = rank_sum(gp + (long long)i * ncta, rows);
                if (threadIdx.x == 0) res[i] = s;
            }
            __syncthreads();
            for (unsigned q = threadIdx.x; q < ncta; q += blockDim.x) gr[(long long)q * RB_SM + i] = res[i];
        }
        cg::this_grid().sync();
        for (int i = threadIdx.x; i < n; i += blockDim.x) res[i] = gr[(long long)crank * RB_SM + i];
        __syncthreads();
        return res;
    }
    __device__ double sum(double v) {
        double a[1] = {v};
        sumk<1>(a);
        return a[0];
    }
    __device__ int any(int flag) { return sum(flag ? 1.0 : 0.0) > 0.0; }
};

}  // namespace rb
