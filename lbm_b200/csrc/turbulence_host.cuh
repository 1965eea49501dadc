// turbulence_host.cuh -- C ABI of the GPU inflow-turbulence generator
// (declaration in include/lbm_b200.h).  Included at the end of api.cu.

#include "turbulence.cuh"

namespace {

// Bytes of the transform buffer a context keeps, unless one group of levels needs
// more: the levels go through it in chunks, so its size does not grow with nrturb,
// and a chunk stays in L2 between the spectrum, the transform and the chain.
constexpr size_t kTurbBufBytes = 64u << 20;

void turb_release(lbm_ctx* c) {
    if (c->turb_planes > 0) cufftDestroy(c->turb_plan);
    cudaFree(c->d_turb_buf);
    cudaFree(c->d_turb_part);
    c->turb_planes = 0;
    c->d_turb_buf = nullptr;
    c->d_turb_part = nullptr;
}

// the transform's plan and buffer for `planes` planes of the context's size, kept
// until the context is destroyed or a call needs another number of planes (making
// them on each call cost 3 to 14 ms)
int turb_workspace(lbm_ctx* c, int planes, int n1, int n2) {
    if (c->turb_planes == planes) return LBM_OK;
    turb_release(c);
    int rc = cuda_check(c, cudaMalloc(&c->d_turb_buf, (size_t)planes * n2 * (n1 / 2 + 1) * sizeof(float2)),
                        "cudaMalloc(turbulence planes)");
    if (rc == LBM_OK)
        rc = cuda_check(c, cudaMalloc(&c->d_turb_part, (size_t)8 * LBM_TURB_MAXBLK * LBM_TURB_NS * sizeof(double)),
                        "cudaMalloc(turbulence sums)");
    int n[2] = {n2, n1};
    if (rc == LBM_OK &&
        cufftPlanMany(&c->turb_plan, 2, n, nullptr, 1, 0, nullptr, 1, 0, CUFFT_C2R, planes) != CUFFT_SUCCESS)
        rc = fail(c, LBM_ERR_CUDA, "inflow_turbulence_compute: cufftPlanMany failed");
    if (rc == LBM_OK) c->turb_planes = planes;
    else turb_release(c);
    return rc;
}

}  // namespace

extern "C" {

int lbm_inflow_turbulence_compute(lbm_ctx* c, float* uu, float* vv, float* ww, float* rr, int32_t nrturb,
                                  uint64_t seed) {
    if (!c) return LBM_ERR_ARG;
    NEED(c, uu); NEED(c, vv); NEED(c, ww);
    if (nrturb < 1) return fail(c, LBM_ERR_ARG, "inflow_turbulence_compute: nrturb must be positive");
    const int ny = c->p.ny, nz = c->p.nz;
    if ((long long)ny * nz < 2) return fail(c, LBM_ERR_ARG, "inflow_turbulence_compute: the (j, k) plane needs 2 cells");
    // m_inflow_turbulence_compute.F90:19-20, 28-32 and m_pseudo2D.F90:61-105: n1 = ny, n2 = nz made even,
    // dx = dy = 1, decorrelation length 10/sqrt(3) in both directions, theta = 0, no mean
    const int n1 = ny + (ny & 1), n2 = nz + (nz & 1);
    const int nf = rr ? 4 : 3;
    const double pi2 = 2.0 * 3.141592653589793;
    const double rx = 10.0 / sqrt(3.0);
    const double deltak = pi2 * pi2 / ((double)n1 * n2);
    const double kappa2 = (pi2 / n1) * (pi2 / n1), lambda2 = (pi2 / n2) * (pi2 / n2);
    const double r1 = sqrt(8.0) / rx, r2 = sqrt(8.0) / rx;   // the reference derives both from rx
    // the sum over the wavenumbers is a product of two one-dimensional sums
    double sum1 = 0.0, sum2 = 0.0;
    for (int l = -n1 / 2 + 1; l <= n1 / 2; ++l) sum1 += exp(-2.0 * (kappa2 * l * l / (r1 * r1)));
    for (int p = -n2 / 2 + 1; p <= n2 / 2; ++p) sum2 += exp(-2.0 * (lambda2 * p * p / (r2 * r2)));
    double summ = sum1 * sum2;
    summ -= 1.0;   // the mean is not sampled
    const double cc = sqrt(1.0 / (deltak * summ));
    TurbSpec s;
    s.n1 = n1;
    s.n2 = n2;
    s.nt = nrturb + 1;
    s.amp = (float)(sqrt(deltak) * cc);
    s.ak = (float)(kappa2 / (r1 * r1));
    s.al = (float)(lambda2 / (r2 * r2));
    s.seed = seed;

    // chunks of whole groups of levels, of about equal length
    const int groups = nrturb / LBM_TURB_B + 1;
    const size_t group_bytes = (size_t)nf * LBM_TURB_B * n2 * (n1 / 2 + 1) * sizeof(float2);
    const int per = (int)std::max<size_t>(1, std::min<size_t>(groups, kTurbBufBytes / group_bytes));
    const int nchunk = (groups + per - 1) / per;
    const int gchunk = (groups + nchunk - 1) / nchunk;
    const int C = gchunk * LBM_TURB_B, planes = nf * C;
    LBM_TRY(turb_workspace(c, planes, n1, n2));
    if (cufftSetStream(c->turb_plan, c->stream) != CUFFT_SUCCESS)
        return fail(c, LBM_ERR_CUDA, "inflow_turbulence_compute: cufftSetStream failed");
    TurbChain ch;
    ch.Y = c->d_turb_buf;
    float* outs[4] = {uu, vv, ww, rr};
    for (int f = 0; f < 4; ++f) ch.o[f] = outs[f];
    ch.part = c->d_turb_part;
    ch.ny = ny;
    ch.nz = nz;
    ch.n2 = n2;
    ch.pitch = 2 * (n1 / 2 + 1);   // an in-place transform leaves its rows at the spectrum's pitch
    ch.C = C;
    ch.nrturb = nrturb;
    // the plane is small (two state buffers of 36 or more elements per row and direction fit the
    // card), so 32-bit indices hold it; about four cells per thread
    const int nblk = std::min(LBM_TURB_MAXBLK, (ny * nz + 4 * LBM_TURB_T - 1) / (4 * LBM_TURB_T));
    const int h = n1 / 2 + 1;
    const dim3 sgrd((unsigned)((n2 * h + 255) / 256), (unsigned)((planes + LBM_TURB_LPT - 1) / LBM_TURB_LPT));
    int rc = LBM_OK;
    for (int g0 = 0; g0 < groups && rc == LBM_OK; g0 += gchunk) {
        const int g1 = std::min(groups, g0 + gchunk);
        ch.t0 = g0 * LBM_TURB_B;
        k_turb_spectrum<<<sgrd, 256, 0, c->stream>>>((float2*)c->d_turb_buf, s, ch.t0, C, planes);
        c->launches++;
        rc = cuda_check(c, cudaGetLastError(), "turbulence spectrum");
        if (rc == LBM_OK &&
            cufftExecC2R(c->turb_plan, reinterpret_cast<cufftComplex*>(c->d_turb_buf), c->d_turb_buf) != CUFFT_SUCCESS)
            rc = fail(c, LBM_ERR_CUDA, "inflow_turbulence_compute: cufftExecC2R failed");
        // sums of the chunk's first group; then each group's levels with the next group's
        // sums; the last group's levels while its planes are still in the buffer
        for (int g = g0 - 1; g < g1 && rc == LBM_OK; ++g) {
            const int ga = g < g0 ? -1 : g, gc = g + 1 < g1 ? g + 1 : -1;
            rc = cuda_check(c, launch_pdl(k_turb_chain, dim3(nblk, nf), dim3(LBM_TURB_T), c->stream, ch, ga, gc),
                            "turbulence levels");
            c->launches++;
        }
    }
    // the caller may read the fields from any stream once this returns
    const int rs = cuda_check(c, cudaStreamSynchronize(c->stream), "inflow_turbulence_compute");
    return rc != LBM_OK ? rc : rs;
}

}  // extern "C"
