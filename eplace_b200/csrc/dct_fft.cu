// dct_fft.cu -- the plan of the fast-transform Poisson solve (fft_kernels.cuh).
#include <new>
#include <string>
#include <vector>

#include "fft.h"

namespace ep {

namespace {

int ilog2_exact(int n) {
    int l = 0;
    while ((1 << l) < n) l++;
    return (1 << l) == n ? l : -1;
}

}  // namespace

int dct_fft_init(DctPlan &p, const std::vector<double> &wx, const std::vector<double> &wy, int fp64,
                 std::string &err) {
    const int nx = p.nx, ny = p.ny;
    const int lx = ilog2_exact(nx), ly = ilog2_exact(ny);
    if (lx < kMinLog || ly < kMinLog || lx > kMaxLog || ly > kMaxLog) {
        err = "the FFT Poisson path needs power-of-two bin counts in [8, 2048]";
        return EP_ERR_UNSUPPORTED;
    }
    FftPlan *f = new (std::nothrow) FftPlan;
    if (!f) {
        err = "out of host memory for the FFT plan";
        return EP_ERR_NOMEM;
    }
    p.fft = f;
    f->lognx = lx;
    f->logny = ly;
    f->fp64 = fp64;
    return fp64 ? FftPasses<double>::init(f, nx, ny, wx, wy, err) : FftPasses<float>::init(f, nx, ny, wx, wy, err);
}

void dct_fft_free(DctPlan &p) {
    FftPlan *f = (FftPlan *)p.fft;
    if (!f) return;
    for (void *d : {f->twx, f->twy, f->qx, f->qy, f->wx, f->wy, f->T, f->X})
        if (d) cudaFree(d);
    delete f;
    p.fft = nullptr;
}

int dct_fft_run(DctPlan &p, const void *rho, void *field, void *phi, const DevScalars *S, cudaStream_t st) {
    const FftPlan *f = (const FftPlan *)p.fft;
    if (f->fp64)
        FftPasses<double>::run(f, p.nx, p.ny, (const double *)rho, (double2 *)field, (double *)phi, S, st);
    else
        FftPasses<float>::run(f, p.nx, p.ny, (const float *)rho, (float2 *)field, (float *)phi, S, st);
    return EP_OK;
}

}  // namespace ep
