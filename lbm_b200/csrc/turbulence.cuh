// turbulence.cuh -- inflow-turbulence fields on the GPU
// (m_inflow_turbulence_compute.F90:3-62 with m_pseudo2D.F90:3-169).
//
// Each level of each field is a 2-D Gaussian random field on the (j, k) plane:
// Fourier amplitudes e(l,p) = exp(-(a11 kappa^2 l^2 + a22 lambda^2 p^2)) with
// uniformly random phases, scaled so the field variance is one
// (m_pseudo2D.F90:96-143), synthesised by a complex-to-real FFT (cuFFT here,
// FFTW there).  The levels 1..nrturb are then chained by the AR(1) relation
// x_t = 0.98 x_(t-1) + sqrt(1 - 0.98^2) x_t and each is normalised to zero mean
// and unit sample standard deviation (m_inflow_turbulence_compute.F90:35-60).
//
// The phases come from SplitMix64 (Steele, Lea and Flood 2014; the finaliser
// of Vigna's splitmix64) applied to a counter built from the seed, the field,
// the level and the wavenumber, instead of the compiler's random_number.  The
// wavenumber columns l = 0 and l = n1/2 are made Hermitian (x(l,-p) =
// conj(x(l,p)), real at the self-conjugate points), so the real transform is
// well defined whatever FFT library runs it.
#pragma once

#include <cstdint>

#include "common.cuh"

namespace lbm {

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    uint64_t z = x + 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

// uniform in [0, 1) with 24 random bits
__host__ __device__ __forceinline__ float unit_uniform(uint64_t seed, uint64_t counter) {
    return (float)(splitmix64(seed ^ splitmix64(counter)) >> 40) * (1.0f / 16777216.0f);
}

struct TurbSpec {
    int n1, n2;          // FFT grid (ny, nz rounded up to even)
    int nt;              // levels of a field, nrturb + 1: the hash counts (field, level) pairs
    float amp;           // sqrt(deltak) * c
    float ak, al;        // a11 kappa^2, a22 lambda^2
    uint64_t seed;
};

// The spectra of the levels [t0, t0 + C) of every field, field-major, plane
// b = field C + (level - t0): X[b][p_idx][l], l = 0..n1/2, p_idx = 0..n2-1
// (p = p_idx, or p_idx - n2 above n2/2 - 1).  Bound by the hash and sincos of
// each value.  A thread keeps one wavenumber and walks LPT planes, so the
// amplitude's exponential and the index arithmetic are paid once per LPT values
// (256 x 256, 303 planes: 92 us with a thread per value).  The phase is 2 pi u
// with u a multiple of 2^-24, so sincospi(2 u) takes it without a rounded 2 pi.
#define LBM_TURB_LPT 8
__global__ void __launch_bounds__(256) k_turb_spectrum(float2* __restrict__ X, TurbSpec s, int t0, int C, int nplanes) {
    const int h = s.n1 / 2 + 1;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= s.n2 * h) return;
    const int pi = m / h, l = m - pi * h;
    int p = pi < s.n2 / 2 ? pi : pi - s.n2;
    // Hermitian columns: the value at -p is the conjugate of the one at p
    const bool herm = (l == 0 || l == s.n1 / 2);
    float sgn = 1.0f;
    bool real_only = false;
    if (herm) {
        if (p < 0 && p != -s.n2 / 2) {
            p = -p;
            sgn = -1.0f;
        }
        real_only = (p == 0 || p == -s.n2 / 2);
    }
    const float mean_off = (l == 0 && p == 0) ? 0.0f : 1.0f;   // lmean = .false.: no mean in any realisation
    const float ee = mean_off * s.amp * expf(-(s.ak * (float)(l * l) + s.al * (float)(p * p)));
    const float ei = real_only ? 0.0f : sgn * ee;
    const uint64_t per_plane = (uint64_t)(s.n2 + 1) * (uint64_t)h;
    const uint64_t base = (uint64_t)(p + s.n2 / 2) * (uint64_t)h + (uint64_t)l;
#pragma unroll 2
    for (int q = 0; q < LBM_TURB_LPT; ++q) {
        const int b = blockIdx.y * LBM_TURB_LPT + q;
        if (b >= nplanes) return;
        const int f = b / C, t = t0 + (b - f * C);
        const uint64_t counter = (uint64_t)(f * s.nt + t) * per_plane + base;
        float sn, cs;
        sincospif(2.0f * unit_uniform(s.seed, counter), &sn, &cs);
        X[(long long)b * s.n2 * h + m] = make_float2(ee * cs, ei * sn);
    }
}

// ---- the AR(1) chain ---------------------------------------------------------------
//
// Level t is o_t = (r_t - mean r_t) / std r_t with r_t = tc o_(t-1) + tn y_t.
// Taken literally each level waits for two sums over the plane of the level
// before it (one block per field did that: 5.2 ms for three fields of 101
// levels at 256 x 256, a serial chain on 3 of 148 SMs).  But every o_t is a
// linear combination of an earlier level o_s and of y_(s+1) .. y_t, so the means
// and deviations of LBM_TURB_B levels follow from the sums and products of
// those LBM_TURB_B + 1 fields, taken in one pass over the plane.  Levels go in
// groups: group g holds the levels 8 g .. 8 g + 7 (level 0 is y_0 itself), and
// one launch applies the chain to group ga and, with the last of its levels
// still in a register, sums the products of group gc = ga + 1.  Launch ga reads
// the block partials that the launch before it wrote.  Sums are in FP64, as the
// means and deviations of the literal form; they are reduced in a fixed order.
#define LBM_TURB_B 8
#define LBM_TURB_T 128                     // threads per block
#define LBM_TURB_MAXBLK 128                // blocks per field: 3 fields stay one wave at 3 blocks per SM
// sums of a group: S(o), S(y_q), S(o o), S(o y_q), S(y_q y_r) q <= r
#define LBM_TURB_NS (2 * (1 + LBM_TURB_B) + LBM_TURB_B * (LBM_TURB_B + 1) / 2)

struct TurbChain {
    const float* Y;      // y of the levels [t0, t0 + C): plane f C + (t - t0), n2 rows of `pitch`
    float* o[4];         // outputs (ny, nz, 0:nrturb)
    double* part;        // block partials of two consecutive groups
    int ny, nz, n2, pitch, C, nrturb, t0;
};

// sum over the 32 lanes of each of 64 values per lane: after the exchange with
// lane ^ 16, 8, 4, 2, 1 a lane holds half as many sums, so it takes 62 exchanges
// instead of 5 x 64; lane i ends with the sums of the values 2 i and 2 i + 1 in
// v[0] and v[1]
__device__ __forceinline__ void warp_sum64(double (&v)[64]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16, half = 32; o > 0; o >>= 1, half >>= 1) {
        const bool hi = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < half; ++q) {
            const double give = hi ? v[q] : v[q + half];
            const double keep = hi ? v[q + half] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
}

__global__ void __launch_bounds__(LBM_TURB_T, 3) k_turb_chain(TurbChain c, int ga, int gc) {
    pdl_enter();
    constexpr int B = LBM_TURB_B, NS = LBM_TURB_NS, T = LBM_TURB_T;
    static_assert(NS <= 64, "warp_sum64 holds 64 sums");
    static_assert(2 * NS <= T, "two threads per sum");
    __shared__ double sum[T];
    __shared__ double wsum[T / 32][64];
    __shared__ float smean[B], sinv[B];
    const int f = blockIdx.y, nblk = gridDim.x, tid = threadIdx.x;
    const float tc = 0.98f, tn = sqrtf(1.0f - 0.98f * 0.98f);
    const int plane = c.ny * c.nz;
    float* out = c.o[f];
    int a0 = 0, na = 0;                    // levels applied: a0 .. a0 + na - 1
    if (ga >= 0) {
        a0 = max(1, B * ga);
        na = min(B * ga + B - 1, c.nrturb) - a0 + 1;
        // the group's sums from the partials of all blocks, two threads per sum
        const double* p = c.part + ((long long)((ga & 1) * 4 + f) * LBM_TURB_MAXBLK) * NS;
        double s = 0.0;
        if (tid < 2 * NS) {
            const int i = tid % NS;
#pragma unroll 16
            for (int b = tid / NS; b < nblk; b += 2) s += p[(long long)b * NS + i];
        }
        sum[tid] = s;
        __syncthreads();
        if (tid < 32) {
            // lane q holds level a0 + q: means, centred products with o and y_r
            const int q = min(tid, B - 1);
            const double n = (double)plane, rn = 1.0 / n;
            auto S = [&](int i) { return sum[i] + sum[NS + i]; };
            const double so = S(0), sy = S(1 + q);
            double G[B];                   // <y_q, y_r>, centred
#pragma unroll
            for (int r = 0; r < B; ++r) {
                const int lo = min(q, r), hi = max(q, r);
                G[r] = S(2 * (1 + B) + lo * B - lo * (lo - 1) / 2 + (hi - lo)) - sy * S(1 + r) * rn;
            }
            double po = S(1 + B + 1 + q) - sy * so * rn;   // <o, y_q>
            double oo = S(1 + B) - so * so * rn;           // <o, o>
            double mo = so * rn;                           // mean of o
            const double dtc = tc, dtn = tn;
#pragma unroll
            for (int t = 0; t < B; ++t) {
                const double pt = __shfl_sync(0xffffffffu, po, t), gtt = __shfl_sync(0xffffffffu, G[t], t);
                const double var = dtc * dtc * oo + 2.0 * dtc * dtn * pt + dtn * dtn * gtt;
                const double inv = 1.0 / sqrt(var / (n - 1.0));
                if (tid == t) {
                    smean[t] = (float)(dtc * mo + dtn * (sy * rn));
                    sinv[t] = (float)inv;
                }
                po = inv * (dtc * po + dtn * G[t]);
                oo = n - 1.0;
                mo = 0.0;
            }
        }
        __syncthreads();
    }
    int c0 = 0, nc = 0;                    // levels summed: c0 .. c0 + nc - 1, after level c0 - 1
    if (gc >= 0) {
        c0 = max(1, B * gc);
        nc = max(0, min(B * gc + B - 1, c.nrturb) - c0 + 1);
    }
    double acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.0;
    const long long ystep = (long long)c.n2 * c.pitch;
    const float* Yf = c.Y + (long long)f * c.C * ystep;
    for (int e = blockIdx.x * T + tid; e < plane; e += nblk * T) {
        const int k = e / c.ny, j = e - k * c.ny;
        const float* y = Yf + (long long)k * c.pitch + j;   // level t0
        float ya[B], yc[B];
#pragma unroll
        for (int q = 0; q < B; ++q) ya[q] = q < na ? y[(a0 + q - c.t0) * ystep] : 0.0f;
#pragma unroll
        for (int q = 0; q < B; ++q) yc[q] = q < nc ? y[(c0 + q - c.t0) * ystep] : 0.0f;
        float o;
        if (gc == 0) {
            o = y[0];                      // level 0 as it is
            out[e] = o;
        } else {
            o = out[(long long)((ga >= 0 ? a0 : c0) - 1) * plane + e];
        }
#pragma unroll
        for (int q = 0; q < B; ++q) {
            if (q >= na) break;
            o = ((tc * o + tn * ya[q]) - smean[q]) * sinv[q];
            out[(long long)(a0 + q) * plane + e] = o;
        }
        if (gc < 0) continue;
        const double d = o;
        acc[0] += d;
        acc[1 + B] += d * d;
        int i = 2 * (1 + B);
#pragma unroll
        for (int q = 0; q < B; ++q) {
            const double yq = yc[q];
            acc[1 + q] += yq;
            acc[2 + B + q] += d * yq;
#pragma unroll
            for (int r = q; r < B; ++r) acc[i++] += yq * (double)yc[r];
        }
    }
    if (gc < 0) return;
    warp_sum64(acc);
    wsum[tid >> 5][2 * (tid & 31)] = acc[0];
    wsum[tid >> 5][2 * (tid & 31) + 1] = acc[1];
    __syncthreads();
    if (tid < NS) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < T / 32; ++w) s += wsum[w][tid];
        c.part[((long long)((gc & 1) * 4 + f) * LBM_TURB_MAXBLK + blockIdx.x) * NS + tid] = s;
    }
}

}  // namespace lbm
