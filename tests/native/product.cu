// prod64_team (rb_product.cuh) on a team of independent CTAs, and the plain loop over k it stands for.
#include "rb_product.cuh"

#include <math.h>

struct Team {
    unsigned crank, ncta;
};

__global__ void __launch_bounds__(256) product(rb::Prod64 a, long long bytes) {
    extern __shared__ __align__(16) unsigned char region[];
    rb::prod64_team(Team{blockIdx.x, gridDim.x}, a, region, bytes);
}

struct Sizes {
    int ni, nk, ncol, nm, nmat, parts, scaled, interleave, sel, pre, ncta;
    long long bytes;  // region per CTA
    double alpha;
};

// Arrays: A, B [nk][ni], X [ncol][nk], ks [nmat][nk], tg [nmat], mat [ncol/nm], selv [nk] (sel 1: the k
// whose selv >= 0) or [ni] (sel 2: the rows), pre and out [ncol][ni].
static rb::Prod64 args(const Sizes &z, const double *A, const double *B, const double *X, const double *ks, const double *tg,
                       const int *mat, const double *selv, const double *pre, double *out) {
    rb::Prod64 a{};
    a.A = A;
    a.B = z.parts == 2 ? B : nullptr;
    a.lda = z.ni;
    a.ldi = 1;
    a.ni = z.ni;
    a.nk = z.nk;
    a.X = X;
    a.sx = 1;
    a.ldx = z.nk;
    a.ncol = z.ncol;
    a.ks = z.scaled ? ks : nullptr;
    a.ksld = z.nk;
    a.tg = z.parts == 2 ? tg : nullptr;
    a.mat = mat;
    a.nm = z.nm;
    a.pre = z.pre ? pre : nullptr;
    a.alpha = z.alpha;
    a.out = out;
    a.so = 1;
    a.ldo = z.ni;
    a.sel = z.sel ? selv : nullptr;
    a.selk = z.sel == 1;
    a.selpos = true;
    a.interleave = z.interleave;
    return a;
}

// The sums as a chain of FMAs in increasing k, part A before part B or (interleave) four of A and four
// of B in turn; `seg` > 0: one part and `seg` values of k at a time, each added to the output before.
extern "C" void product_loop(const Sizes *z, const double *A, const double *B, const double *X, const double *ks, const double *tg,
                             const int *mat, const double *selv, const double *pre, double *out, int seg) {
    for (long long c = 0; c < z->ncol; c++)
        for (int i = 0; i < z->ni; i++) {
            if (z->sel == 2 && !(selv[i] >= 0)) continue;
            const int m = mat[c / z->nm];
            auto term = [&](int part, int k, double acc) {
                if (z->sel == 1 && !(selv[k] >= 0)) return acc;
                const double s = part ? tg[m] : (z->scaled ? ks[(long long)m * z->nk + k] : 1.0);
                return fma(s * X[c * z->nk + k], (part ? B : A)[(long long)k * z->ni + i], acc);
            };
            double o = z->pre ? pre[c * z->ni + i] : 0.0;
            if (z->interleave && z->parts == 2 && !seg) {
                double acc = 0.0;
                for (int k0 = 0; k0 < z->nk; k0 += 4)
                    for (int p = 0; p < 2; p++)
                        for (int k = k0; k < k0 + 4 && k < z->nk; k++) acc = term(p, k, acc);
                o = fma(z->alpha, acc, o);
            } else {
                double acc = 0.0;
                for (int p = 0; p < z->parts; p++)
                    for (int k = 0; k < z->nk; k++) {
                        if (seg && k % seg == 0 && (p || k)) {
                            o = fma(z->alpha, acc, o);
                            acc = 0.0;
                        }
                        acc = term(p, k, acc);
                    }
                o = fma(z->alpha, acc, o);
            }
            out[c * z->ni + i] = o;
        }
}

// values of k of one piece of an operator cut along k (0: not cut)
extern "C" int product_seg(const Sizes *z) {
    if (rb::prod_blocks(z->ni, z->nk, z->parts, z->bytes)) return 0;
    int n = 1;
    while (!rb::prod_blocks(z->ni, (z->nk + n - 1) / n, 1, z->bytes)) n++;
    return (z->nk + n - 1) / n;
}

extern "C" int product_device(const Sizes *z, const double *A, const double *B, const double *X, const double *ks, const double *tg,
                              const int *mat, const double *selv, const double *pre, double *out) {
    const size_t no = (size_t)z->ncol * z->ni, nx = (size_t)z->ncol * z->nk, nA = (size_t)z->ni * z->nk, nks = (size_t)z->nmat * z->nk;
    const size_t nsel = z->sel == 2 ? z->ni : z->nk, nmt = (z->ncol + z->nm - 1) / z->nm;
    const size_t n = 2 * nA + nx + nks + z->nmat + nsel + 2 * no + 16;
    double *d = nullptr;
    int *dm = nullptr;
    cudaError_t e = cudaMalloc(&d, n * 8);
    if (e == cudaSuccess) e = cudaMalloc(&dm, nmt * 4);
    double *p = d;
    auto put = [&](const double *h, size_t k) {
        double *q = p;
        p += (k + 1) & ~(size_t)1;
        if (e == cudaSuccess && h) e = cudaMemcpy(q, h, k * 8, cudaMemcpyHostToDevice);
        return q;
    };
    double *dA = put(A, nA), *dB = put(B, nA), *dX = put(X, nx), *dk = put(ks, nks), *dt = put(tg, z->nmat), *ds = put(selv, nsel);
    double *dp = put(pre, no), *dout = put(out, no);
    if (e == cudaSuccess) e = cudaMemcpy(dm, mat, nmt * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(product, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)z->bytes);
    if (e == cudaSuccess) {
        product<<<z->ncta, 256, z->bytes>>>(args(*z, dA, dB, dX, dk, dt, dm, ds, dp, dout), z->bytes);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, no * 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(dm);
    return (int)e;
}
