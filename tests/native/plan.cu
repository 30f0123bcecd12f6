// Host side of the 3D octant sweep's rule and offsets (rb_sweep_oct.cuh) for a 3D one-moment problem,
// and of the team size of a launch (rb_launch.cuh).
#include "rb_launch.cuh"
#include "rb_solve.cuh"

static DevProblem problem(int nx, int ny, int nz, int nd, int csd) {
    DevProblem P{};
    P.ndims = 3;
    P.nx = nx;
    P.ny = ny;
    P.nz = nz;
    P.ncell = (long long)nx * ny * nz;
    P.nd = nd;
    P.csd = csd;
    P.nm5 = P.nm4 = P.nfmax = P.nmf[0] = P.nmf[1] = P.nmf[2] = 1;
    return P;
}
extern "C" int plan_oct3d_ok(int nx, int ny, int nz, int nd, int csd, int ncta, int mixed) {
    return rb::oct3d_ok(problem(nx, ny, nz, nd, csd), ncta, 200 << 10, mixed);
}
extern "C" long long plan_oct_offset(int nx, int ny, int nz, int nd, int f, int qy, int qz, int n) {
    return rb::oct_offset(problem(nx, ny, nz, nd, 0), f & 1, f & 2, f & 4, qy, qz, n);
}
// n equal problems of 200 cells a side, 16 directions, closures of order `order`
extern "C" int plan_cluster(int ndims, int order, int csd, int n, int cluster, int mode) {
    DevProblem P{};
    P.ndims = ndims;
    P.local1d = 1;
    P.nx = 200;
    P.nd = P.np = 16;
    P.nmat = 2;
    P.csd = csd;
    P.nmf[0] = csd ? order : 1;
    P.nm4 = csd ? order : 1;
    P.nm5 = csd ? order * order : order;
    P.nphi = (long long)P.np * P.nm5 * P.nx;
    P.nstate = P.nphi + 2 * 8 * P.nmf[0];
    const std::vector<const DevProblem *> hs(n, &P);
    return choose_cluster(hs, cluster, mode, 148, 190 << 10);
}
