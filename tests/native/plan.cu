// Host side of the 3D octant sweep's rule and offsets (rb_sweep_oct.cuh) for a 3D one-moment problem.
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
