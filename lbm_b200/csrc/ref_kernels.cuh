// ref_kernels.cuh -- per-call kernels on the reference layout
// f(nl,0:nx+1,0:ny+1,0:nz+1) (l fastest), one per reference subroutine.
//
// Cell-wise kernels stage runs of cells (nl contiguous values each) through shared
// memory, so the global reads and writes are coalesced even though each cell's nl
// populations are contiguous; the per-cell math reads the staged values with an odd
// stride (nl = 19 or 27), free of bank conflicts for FP32.  postcoll and macrovars walk
// tiles of 64 or 128 cells that pass over row ends, the next one under way
// (ref_tiles.cuh); the others take a chunk of 128 cells of a row.
//
// Every kernel takes the arithmetic type R as a template argument: float for
// the reference's default build, double for its DP build (the _f64 entry
// points), where -r8 makes every real, tiny() and eps double precision.
#pragma once

#include "boundary.cuh"
#include "collide.cuh"
#include "ref_tiles.cuh"

namespace lbm {


// Equilibrium offsets feq_l - w_l (m_fequil3_kernel.F90:58-113 in closed form).
template <int Q, typename R>
__device__ __forceinline__ void equilibrium(R (&fe)[Q], R drho, R rho, R ux, R uy, R uz, bool cubic) {
    const R usq = ux * ux + uy * uy + uz * uz;
    const R R45 = R(4.5) * rho;
    const R R45o = cubic ? R45 : R(0.0);
    const R A0 = drho - R(1.5) * rho * usq;
    const R B0 = R(3.0) * rho - (cubic ? R45 * usq : R(0.0));
    fe[0] = lat_w<Q, R>(0) * A0;
#pragma unroll
    for (int l = 1; l < Q; l += 2) {
        const R w = lat_w<Q, R>(l);
        const R cu = cdot(lat_cx(l), lat_cy(l), lat_cz(l), ux, uy, uz);
        const R cu2 = cu * cu;
        const R E = w * (A0 + R45 * cu2);
        const R O = w * cu * (B0 + R45o * cu2);
        fe[l] = E + O;
        fe[l + 1] = E - O;
    }
}

// Regularized non-equilibrium R(fneq) from a2 = sum H2 fneq (all l, including rest).
template <int Q, typename R>
__device__ __forceinline__ void regularized(R (&out)[Q], const MomentsT<R>& m, R ux, R uy, R uz) {
    const R third = R(1.0) / R(3.0);
    const R axx = m.pxx - m.s0 * third, ayy = m.pyy - m.s0 * third, azz = m.pzz - m.s0 * third;
    const R axy = m.pxy, axz = m.pxz, ayz = m.pyz;
    const R tr = axx + ayy + azz;
    const R vx = axx * ux + axy * uy + axz * uz;
    const R vy = axy * ux + ayy * uy + ayz * uz;
    const R vz = axz * ux + ayz * uy + azz * uz;
    out[0] = lat_w<Q, R>(0) * R(4.5) * (-tr * third);
#pragma unroll
    for (int l = 1; l < Q; l += 2) {
        const int cx = lat_cx(l), cy = lat_cy(l), cz = lat_cz(l);
        const R w = R(4.5) * lat_w<Q, R>(l);
        const R cu = cdot(cx, cy, cz, ux, uy, uz);
        R cac = R(0);
        macc(cac, cx * cx, axx);
        macc(cac, cy * cy, ayy);
        macc(cac, cz * cz, azz);
        macc(cac, cx * cy, R(2.0) * axy);
        macc(cac, cx * cz, R(2.0) * axz);
        macc(cac, cy * cz, R(2.0) * ayz);
        const R cau = cdot(cx, cy, cz, vx, vy, vz);
        const R E = w * (cac - tr * third);
        const R O = w * (cu * (R(3.0) * cac - tr) - R(2.0) * cau);
        out[l] = E + O;
        out[l + 1] = E - O;
    }
}

// Row-chunk staging: cells [i0, i0+n) of row (j,k), n <= 128.
#define TILE_ILP 8
template <int Q, typename R>
__device__ __forceinline__ void tile_load(R* __restrict__ sm, const R* __restrict__ f, long long cell0, int n) {
    // TILE_ILP independent loads in flight per thread before their shared-memory stores
    const R* src = f + cell0 * Q;
    const int m = n * Q, step = blockDim.x * TILE_ILP;
    for (int e0 = threadIdx.x; e0 < m; e0 += step) {
        R v[TILE_ILP];
#pragma unroll
        for (int u = 0; u < TILE_ILP; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < m) v[u] = src[e];
        }
#pragma unroll
        for (int u = 0; u < TILE_ILP; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < m) sm[e] = v[u];
        }
    }
}
template <int Q, typename R>
__device__ __forceinline__ void tile_store(const R* __restrict__ sm, R* __restrict__ f, long long cell0, int n) {
    R* dst = f + cell0 * Q;
    const int m = n * Q;
    for (int e = threadIdx.x; e < m; e += blockDim.x) dst[e] = sm[e];
}

// fequil3: feq on interior cells (m_fequil3_kernel.F90:7-123)
template <int Q, typename R = float>
__global__ void __launch_bounds__(128) k_ref_fequil3(R* feq, const R* rho, const R* u, const R* v,
                                                     const R* w, RefGrid g, int ibgk) {
    __shared__ R sm[128 * Q];
    const int i0 = blockIdx.x * 128 + 1, j = blockIdx.y + 1, k = blockIdx.z + 1;
    const int n = min(128, g.nx + 1 - i0);
    const int t = threadIdx.x;
    if (n <= 0) return;
    if (t < n) {
        const long long c = g.cell(i0 + t, j, k);
        R fe[Q];
        equilibrium<Q>(fe, rho[c] - R(1.0), rho[c], u[c], v[c], w[c], ibgk == 3);
#pragma unroll
        for (int l = 0; l < Q; ++l) sm[t * Q + l] = fe[l] + lat_w<Q, R>(l);
    }
    __syncthreads();
    tile_store<Q>(sm, feq, g.cell(i0, j, k), n);
}

// Shared memory and resident blocks of the tiled kernels: two tile buffers with
// `scalars` values per cell each; as many blocks as fit an SM, up to a cap on
// their registers.
// T: postcoll reads, computes and writes between three barriers, so more, smaller blocks
// serve it.  us in tiles of 64 and of 128 cells:
//              128x64x64     192x96x96      256x128x128    512x128x128
//   D3Q27 FP32 32.9  33.9    90.9  99.8     196.0 207.5    365.0 375.1
//   D3Q27 FP64 52.8  60.2    155.4 180.5    334.9 371.5    642.5 681.6
//   D3Q19 FP64 39.4  42.0    107.9 116.6    241.8 253.9    477.5 472.4
//   D3Q19 FP32 29.1  27.4    70.9  74.2     165.8 173.8    300.3 307.8
// D3Q19 FP32 was set to 128 on the first column alone, the one in which 64 loses; larger
// grids would gain 2 to 5% from 64.  macrovars is within 2% (3% for D3Q27 FP32
// 512x128x128) either way.
template <int Q, typename R>
struct PostcollTile {
    static constexpr int T = (sizeof(R) == 4 && Q == 19) ? 128 : 64;
    static constexpr int SC = 5;                                   // rho, u, v, w, tau
    static constexpr int STAGE = CellTile<Q, R, T>::BUF + SC * T;   // elements of one of the two stages
    static constexpr size_t SMEM = 2 * STAGE * sizeof(R);
    static constexpr int BLOCKS = sizeof(R) == 4 ? (Q == 27 ? 12 : 7) : (Q == 27 ? 6 : 8);
};
template <int Q, typename R>
struct MacroTile {
    static constexpr int T = 128;
    static constexpr int STAGE = CellTile<Q, R, T>::BUF;
    static constexpr size_t SMEM = 2 * STAGE * sizeof(R);
    static constexpr int BLOCKS = sizeof(R) == 4 ? (Q == 27 ? 7 : 10) : (Q == 27 ? 4 : 5);
};

// postcoll: collide interior cells in place with the given moments (m_postcoll_kernel.F90:7-255)
template <int Q, typename R = float>
__global__ void __launch_bounds__(PostcollTile<Q, R>::T, PostcollTile<Q, R>::BLOCKS)
    k_ref_postcoll(R* f, R* tau, const R* rho, const R* u, const R* v, const R* w, const R* abl, RefGrid g,
                   CollideParamsT<R> cp, unsigned tp, unsigned ntiles) {
    using P = PostcollTile<Q, R>;
    constexpr int T = P::T;
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ unsigned cells[T / 32];
    R* sm = reinterpret_cast<R*>(raw);
    const int tid = threadIdx.x;
    auto fetch = [&](unsigned t, int b) {
        const TileAt a = tile_at<false, T>(g, t, tp);
        tile_fetch<Q, T>(sm + b * P::STAGE, f, a.c0, a.n);
        if (tid < a.n) {
            R* s = sm + b * P::STAGE + CellTile<Q, R, T>::BUF + tid;
            const long long c = a.c0 + tid;
            cp_async_elem(s, rho + c);
            cp_async_elem(s + T, u + c);
            cp_async_elem(s + 2 * T, v + c);
            cp_async_elem(s + 3 * T, w + c);
            cp_async_elem(s + 4 * T, tau + c);
        }
    };
    fetch(blockIdx.x, 0);
    cp_async_commit();
    int b = 0;
    for (unsigned t = blockIdx.x; t < ntiles; t += gridDim.x, b ^= 1) {
        if (t + gridDim.x < ntiles) fetch(t + gridDim.x, b ^ 1);
        cp_async_commit();
        const TileAt a = tile_at<false, T>(g, t, tp);
        const unsigned i = (a.q0 + tid) % (unsigned)(g.nx + 2);
        const bool inner = tid < a.n && i >= 1 && i <= (unsigned)g.nx;
        const unsigned mask = __ballot_sync(0xffffffffu, inner);
        if ((tid & 31) == 0) cells[tid >> 5] = mask;
        cp_async_wait<1>();
        __syncthreads();
        R* tile = sm + b * P::STAGE;
        if (inner) {
            R* s = tile + phase_of(f + a.c0 * Q) + tid * Q;
            const R* sc = tile + CellTile<Q, R, T>::BUF + tid;
            R fp[Q];
#pragma unroll
            for (int l = 0; l < Q; ++l) fp[l] = s[l] - lat_w<Q, R>(l);
            const MomentsT<R> m = moments<Q>(fp);
            const R r = sc[0];
            TurbInT<R> tb;
            tb.on = false;
            tb.dux = tb.duy = tb.duz = R(0);
            const R tnew = collide<Q>(fp, m, r - R(1.0), r, sc[T], sc[2 * T], sc[3 * T], cp,
                                      abl ? abl[a.k - 1] : R(0.0), sc[4 * T], false, tb);
            if (cp.ivreman) tau[a.c0 + tid] = tnew;
#pragma unroll
            for (int l = 0; l < Q; ++l) s[l] = fp[l] + lat_w<Q, R>(l);
        }
        const bool whole = __syncthreads_and(inner);
        tile_put<Q, T>(tile, f, a.c0, a.n, cells, whole);
        __syncthreads();
    }
}

// drift: f(l,i,j,k) = feq(l,i-cx,j-cy,k-cz) over interior cells
// (m_drift_kernel.F90:33-42).
//
// A direction's values lie nl elements apart, so gathering them from global
// memory takes one 32-byte sector per element (347 us for D3Q27 256x128x128
// FP32, 2.6 TB/s of the bytes it must move; 140 us for D3Q19 192x96x96 FP64).
// Instead a block owns TJ rows of NI cells and marches along k with a ring of
// planes of its rows and their neighbours in shared memory: the three that an
// output plane needs and the next ones, still arriving.  A source row crosses L2
// about 1.6 times ((TJ+2)/TJ (NI+2)/NI) instead of nine, all copies are whole
// 16-byte words, and a thread writes one direction: its source sits at a fixed
// distance.
//
// A row of the ring starts at the phase its global address has in a word
// (ref_tiles.cuh): the row stride rs equals the global one modulo a word, and a
// plane is placed at its own phase.  The words at a row's ends bring up to a
// word of its neighbours along; only at the two ends of the array, where a word
// could reach past it, do they move element by element.
template <int Q, typename R>
struct DriftTile {
    static constexpr int TJ = (sizeof(R) == 8 && Q == 27) ? 3 : 4;
    static constexpr int NI = 128 / (int)sizeof(R);            // cells of a row: 32 FP32, 16 FP64
    static constexpr int SLOTS = Q == 27 ? 5 : 6;              // planes of the ring: two blocks fill an SM
    static constexpr int AHEAD = SLOTS - 3;                    // planes under way
    static constexpr int LANES = 16;                           // cells per pass of a block
    static constexpr int T = Q * LANES;                        // a thread per (cell, direction)
    static constexpr int V = word_elems<R>();
    static constexpr int ROW = (NI + 2) * Q;                   // elements of a row, at most
    static constexpr int WORDS = (ROW + 2 * (V - 1)) / V;      // words a row may touch
    static constexpr int RS = (WORDS + 2) * V;                 // row stride, at most
    static constexpr int PS = (TJ + 2) * RS + V;               // plane stride
    static constexpr size_t SMEM = (size_t)SLOTS * PS * sizeof(R);
    static constexpr int BLOCKS = 2;
    static_assert(BLOCKS * (SMEM + 1024) <= 228 * 1024, "the blocks fit an SM");
};
struct DriftShape {
    int ni;        // cells of a row chunk
    int ks;        // planes of a k segment
    int rs;        // row stride of the ring: room for a row, congruent to the global stride
};
template <int Q, typename R>
int drift_row_stride(const RefGrid& g) {
    using D = DriftTile<Q, R>;
    return (D::WORDS + 1) * D::V + (int)(((long long)(g.nx + 2) * Q) % D::V);
}
// rows of g.nx cells, g.ny rows, g.nz planes of an array with one ghost cell at every end
template <int Q, typename R>
DriftShape drift_shape(const RefGrid& g, int slots) {
    using D = DriftTile<Q, R>;
    DriftShape d;
    const int nch = (g.nx + D::NI - 1) / D::NI;
    d.ni = (g.nx + nch - 1) / nch;
    d.rs = drift_row_stride<Q, R>(g);
    // segments of k: a block takes about ks + 4 plane times (two extra planes and the
    // first ones' latency); `slots` blocks run at a time
    const long long columns = (long long)nch * ((g.ny + D::TJ - 1) / D::TJ);
    long long best = -1;
    d.ks = g.nz;
    for (int ns = 1; ns <= g.nz && ns <= 64; ++ns) {
        const int ks = (g.nz + ns - 1) / ns;
        const long long cost = (columns * ((g.nz + ks - 1) / ks) + slots - 1) / slots * (ks + 4);
        if (best < 0 || cost < best) {
            best = cost;
            d.ks = ks;
        }
    }
    return d;
}

template <int Q, typename R = float>
__global__ void __launch_bounds__(DriftTile<Q, R>::T, DriftTile<Q, R>::BLOCKS)
    k_ref_drift(R* __restrict__ f, const R* __restrict__ feq, RefGrid g, DriftShape d) {
    using D = DriftTile<Q, R>;
    constexpr int V = D::V, TJ = D::TJ;
    constexpr int LOADS = ((TJ + 2) * D::WORDS + D::T - 1) / D::T;   // words a thread copies per plane
    extern __shared__ __align__(16) unsigned char raw[];
    R* sm = reinterpret_cast<R*>(raw);
    const int tid = threadIdx.x;
    // grid: x over the chunks of a row, then the row tiles; y over the k segments
    const int nch = (g.nx + d.ni - 1) / d.ni, jt = blockIdx.x / nch;
    const int i0 = (blockIdx.x - jt * nch) * d.ni + 1, j0 = jt * TJ + 1, k0 = blockIdx.y * d.ks + 1;
    const int ni = min(d.ni, g.nx + 1 - i0), nj = min(TJ, g.ny + 1 - j0), k1 = min(k0 + d.ks, g.nz + 1);
    if (ni <= 0 || nj <= 0 || k0 >= k1) return;
    const int np = k1 - k0;
    const long long rowg = (long long)(g.nx + 2) * Q, planeg = rowg * (g.ny + 2);
    const R* src = feq + g.cell(i0 - 1, j0 - 1, k0 - 1) * Q;    // first element of plane 0
    const int len = (ni + 2) * Q, ph0 = phase_of(src);
    // a block whose first or last row is the array's
    const bool ends = (i0 == 1 && j0 == 1 && k0 == 1) || (i0 + ni > g.nx && j0 + nj > g.ny && k1 > g.nz);
    // the words this thread copies of each plane: row and word within the row
    int lr[LOADS], lw[LOADS];
#pragma unroll
    for (int q = 0; q < LOADS; ++q) {
        const int e = tid + q * D::T;
        lr[q] = e / D::WORDS;
        lw[q] = e - lr[q] * D::WORDS;
    }
    // plane p (k = k0 - 1 + p) into ring slot `slot`
    auto load_plane = [&](int p, int slot) {
        const R* s = src + p * planeg;
        const int at = slot * D::PS + phase_of(s);
#pragma unroll
        for (int q = 0; q < LOADS; ++q) {
            if (lr[q] >= nj + 2) break;
            const R* row = s + lr[q] * rowg;
            const int o = at + lr[q] * d.rs, ph = o % V;        // element 0 of the row, and its phase
            if (ends) run_load_word(sm + (o - ph), row, ph, len, lw[q]);
            else if (lw[q] * V < ph + len) cp_async16(sm + (o - ph) + lw[q] * V, row - ph + lw[q] * V);
        }
    };
#pragma unroll
    for (int p = 0; p < 2 + D::AHEAD; ++p) {
        if (p < np + 2) load_plane(p, p);
        cp_async_commit();
    }
    const int l = tid % Q;
    const int cz = c_cz[l];
    const int from = (1 - c_cy[l]) * d.rs + (1 - c_cx[l]) * Q + tid;
    R* dst = f + g.cell(i0, j0, k0) * Q + tid;
    const int n = ni * Q;
    int slot = 1, next = 2 + D::AHEAD;                          // slots of the planes p + 1 and p + 2 + AHEAD
    for (int p = 0; p < np; ++p) {                              // output plane k0 + p = plane p + 1
        cp_async_wait<D::AHEAD - 1>();
        __syncthreads();                                        // planes p .. p+2 are here; all are past plane p-1
        if (p + 2 + D::AHEAD < np + 2) load_plane(p + 2 + D::AHEAD, next);
        cp_async_commit();
        int at = slot - cz;
        at += at < 0 ? D::SLOTS : (at >= D::SLOTS ? -D::SLOTS : 0);
        const R* s = sm + at * D::PS + (int)((ph0 + (p + 1 - cz) * planeg) & (V - 1)) + from;
#pragma unroll
        for (int r = 0; r < TJ; ++r) {
            if (r >= nj) break;
#pragma unroll
            for (int m = 0; m < D::NI / D::LANES; ++m)
                if (tid + m * D::T < n) dst[r * rowg + m * D::T] = s[r * d.rs + m * D::T];
        }
        dst += planeg;
        slot = slot + 1 == D::SLOTS ? 0 : slot + 1;
        next = next + 1 == D::SLOTS ? 0 : next + 1;
    }
}

// macrovars over the ghost-inclusive grid, summation order of m_macrovars_kernel.F90:35-49
template <int Q, typename R = float>
__global__ void __launch_bounds__(MacroTile<Q, R>::T, MacroTile<Q, R>::BLOCKS)
    k_ref_macrovars(R* rho, R* u, R* v, R* w, const R* f, RefGrid g, unsigned ntiles) {
    using P = MacroTile<Q, R>;
    constexpr int T = P::T;
    extern __shared__ __align__(16) unsigned char raw[];
    R* sm = reinterpret_cast<R*>(raw);
    const int tid = threadIdx.x;
    auto fetch = [&](unsigned t, int b) {
        const TileAt a = tile_at<true, T>(g, t, 0);
        tile_fetch<Q, T>(sm + b * P::STAGE, f, a.c0, a.n);
    };
    fetch(blockIdx.x, 0);
    cp_async_commit();
    int b = 0;
    for (unsigned t = blockIdx.x; t < ntiles; t += gridDim.x, b ^= 1) {
        if (t + gridDim.x < ntiles) fetch(t + gridDim.x, b ^ 1);
        cp_async_commit();
        const TileAt a = tile_at<true, T>(g, t, 0);
        cp_async_wait<1>();
        __syncthreads();
        if (tid < a.n) {
            const R* s = sm + b * P::STAGE + phase_of(f + a.c0 * Q) + tid * Q;
            R tr = R(0), tu = R(0), tv = R(0), tw = R(0);
#pragma unroll
            for (int l = 0; l < Q; ++l) {
                const R tf = s[l];
                tr = tr + tf;
                macc(tu, lat_cx(l), tf);
                macc(tv, lat_cy(l), tf);
                macc(tw, lat_cz(l), tf);
            }
            const R inv = R(1.0) / tr;
            const long long c = a.c0 + tid;
            rho[c] = tr;
            u[c] = tu * inv;
            v[c] = tv * inv;
            w[c] = tw * inv;
        }
        __syncthreads();
    }
}

// regularization: f = R(f - feq) on interior cells (m_regularization_kernel.F90:6-122)
template <int Q, typename R = float>
__global__ void __launch_bounds__(128) k_ref_regularization(R* f, const R* feq, const R* u,
                                                            const R* v, const R* w, RefGrid g) {
    __shared__ R sm[128 * Q];
    const int i0 = blockIdx.x * 128 + 1, j = blockIdx.y + 1, k = blockIdx.z + 1;
    const int n = min(128, g.nx + 1 - i0);
    const int t = threadIdx.x;
    if (n <= 0) return;
    tile_load<Q>(sm, f, g.cell(i0, j, k), n);
    __syncthreads();
    if (t < n) {
        const long long c = g.cell(i0 + t, j, k);
        R fn[Q];
#pragma unroll
        for (int l = 0; l < Q; ++l) fn[l] = sm[t * Q + l] - feq[c * Q + l];
        const MomentsT<R> m = moments<Q>(fn);
        R out[Q];
        regularized<Q>(out, m, u[c], v[c], w[c]);
#pragma unroll
        for (int l = 0; l < Q; ++l) sm[t * Q + l] = out[l];
    }
    __syncthreads();
    tile_store<Q>(sm, f, g.cell(i0, j, k), n);
}

// vreman: tau from a non-equilibrium f with the standalone guards
// (alphamag and beta start at 1e-5, no ablvisc; m_vreman_kernel.F90:47-91)
template <int Q, typename R = float>
__global__ void __launch_bounds__(128) k_ref_vreman(const R* f, R* tau, RefGrid g, CollideParamsT<R> cp) {
    __shared__ R sm[128 * Q];
    const int i0 = blockIdx.x * 128 + 1, j = blockIdx.y + 1, k = blockIdx.z + 1;
    const int n = min(128, g.nx + 1 - i0);
    const int t = threadIdx.x;
    if (n <= 0) return;
    tile_load<Q>(sm, f, g.cell(i0, j, k), n);
    __syncthreads();
    if (t < n) {
        R fn[Q];
#pragma unroll
        for (int l = 0; l < Q; ++l) fn[l] = sm[t * Q + l];
        const MomentsT<R> m = moments<Q>(fn);
        const R third = R(1.0) / R(3.0);
        const R axx = m.pxx - m.s0 * third, ayy = m.pyy - m.s0 * third, azz = m.pzz - m.s0 * third;
        const R axy = m.pxy, axz = m.pxz, ayz = m.pyz;
        const R g0 = R(0.00001);
        const R amag = g0 + (axx * axx + ayy * ayy + azz * azz + R(2.0) * (axy * axy + axz * axz + ayz * ayz));
        const R b11 = g0 + axx * axx + axy * axy + axz * axz;
        const R b22 = g0 + axy * axy + ayy * ayy + ayz * ayz;
        const R b33 = g0 + axz * axz + ayz * ayz + azz * azz;
        const R b12 = g0 + axx * axy + axy * ayy + axz * ayz;
        const R b13 = g0 + axx * axz + axy * ayz + axz * azz;
        const R b23 = g0 + axy * axz + ayy * ayz + ayz * azz;
        const R bb = b11 * b22 - b12 * b12 + b11 * b33 - b13 * b13 + b22 * b33 - b23 * b23;
        const R tt = bb / amag;
        const R nut = (tt > cp.eps) ? cp.cvre * real_sqrt(tt) : R(0.0);
        tau[g.cell(i0 + t, j, k)] = R(3.0) * (cp.kinevisc + nut) + R(0.5);
    }
}

// compute_fneq / compute_f: elementwise over every element, ghosts included
template <typename R = float>
__global__ void k_ref_axpy(R* f, const R* feq, long long n, int sgn) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        f[e] = (sgn > 0) ? (feq[e] + f[e]) : (f[e] - feq[e]);
}

// solids: swap pairs (l,l+1), l = 2,4,..,nl-1 (1-based) at blanked interior cells (m_solids.F90:24-36).
// A block reads 1024 mask entries in 16-byte words (its first and last ones
// element by element), lists the blanked interior cells among them, and swaps
// their pairs with a thread per pair, so that a cell's values move together
// (a thread per cell walks 108 bytes by itself: 24 us for 256x128x128 with 16 boxes).
#define SOLID_CELLS 1024
template <int Q, typename R = float>
__global__ void __launch_bounds__(256) k_ref_solids(R* f, const int32_t* blank, RefGrid g) {
    __shared__ int count;
    __shared__ int list[SOLID_CELLS];
    const long long n = g.ncell();
    const long long e0 = (long long)blockIdx.x * SOLID_CELLS - phase_of(blank);   // first cell of the block
    const long long e = e0 + threadIdx.x * 4;
    if (threadIdx.x == 0) count = 0;
    int m[4] = {0, 0, 0, 0};
    if (e >= 0 && e + 4 <= n) {
        const int4 q = *reinterpret_cast<const int4*>(blank + e);
        m[0] = q.x; m[1] = q.y; m[2] = q.z; m[3] = q.w;
    } else {
#pragma unroll
        for (int v = 0; v < 4; ++v)
            if (e + v >= 0 && e + v < n) m[v] = blank[e + v];
    }
    if (!__syncthreads_or(m[0] | m[1] | m[2] | m[3])) return;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        if (m[v] == 0) continue;
        const long long c = e + v, row = c / (g.nx + 2), k = row / (g.ny + 2);
        const int i = (int)(c - row * (g.nx + 2)), j = (int)(row - k * (g.ny + 2));
        if (i >= 1 && i <= g.nx && j >= 1 && j <= g.ny && k >= 1 && k <= g.nz)
            list[atomicAdd(&count, 1)] = threadIdx.x * 4 + v;
    }
    __syncthreads();
    constexpr int NP = Q / 2;
    const int work = count * NP;
    for (int w = threadIdx.x; w < work; w += 256) {
        const int cell = w / NP, q = w - cell * NP;
        R* p = f + (e0 + list[cell]) * Q + 1 + 2 * q;
        const R x = p[0], y = p[1];
        p[0] = y;
        p[1] = x;
    }
}

// ---- boundarycond on the reference layout ------------------------------------------
// The kernels of boundary.cuh give a thread a cell (or one direction of cells that
// lie nl elements apart), which suits a structure of arrays.  Here l is fastest,
// so consecutive threads take consecutive directions of a cell.

// the periodic copies of one axis (m_boundary_{i,j,k}_periodic_kernel.F90): the
// ghost planes 0 and n+1 from the planes n and 1.  A thread per element of a
// plane's contiguous pieces (axis 0: a cell, 1: a row, 2: the whole plane).
// Grid: x over a piece's elements (axis 0: over the rows' cells), y over the planes k.
template <typename R>
__global__ void __launch_bounds__(256) k_ref_periodic(R* __restrict__ f, RefGrid g, int axis) {
    const long long row = (long long)(g.nx + 2) * g.nl, plane = row * (g.ny + 2);
    const long long e = (long long)blockIdx.x * 256 + threadIdx.x;
    long long at, step;
    int n;
    if (axis == 0) {
        const long long j = e / g.nl;
        if (j > g.ny + 1) return;
        at = j * row + (e - j * g.nl) + blockIdx.y * plane;
        step = g.nl;
        n = g.nx;
    } else if (axis == 1) {
        if (e >= row) return;
        at = e + blockIdx.y * plane;
        step = row;
        n = g.ny;
    } else {
        if (e >= plane) return;
        at = e;
        step = plane;
        n = g.nz;
    }
    R* p = f + at;
    const R lo = p[n * step], hi = p[step];
    p[0] = lo;
    p[(n + 1) * step] = hi;
}

// closed faces of one axis: k_closed of boundary.cuh with a thread per (outgoing
// direction, cell), which takes the two opposite faces.  wrap (periodic j): a source
// row 0 or ny+1 is read as row ny or 1, so the periodic j copy that comes before it
// in m_boundarycond.F90 need not run.  Bound by latency and issue: a face has 9
// (D3Q27) or 5 (D3Q19) outgoing directions, a constant to divide by, and a direction's
// table entry holds all that depends on it; two cells' loads are under way at once.
// k faces of D3Q27 FP32 256x128x128: 11.6 us (13.3 with a thread per cell, 14.9 with a
// face per thread, a run-time divisor and byte tables); D3Q19 8.1 (8.7, 11.3), FP64
// 192x96x96 6.9 (8.8, 9.2).
template <int Q>
struct ClosedPairs {
    static constexpr int N = Q == 27 ? 9 : 5;   // outgoing directions of a face
};
struct ClosedPair {
    long long d;   // elements from the ghost cell's first value to the source value
    int l, m, cy, pad;
};
template <int Q, typename R>
__global__ void __launch_bounds__(128) k_ref_closed(R* f1, const R* f2, RefGrid g, int axis, FacePairs lo, FacePairs hi, int wrap) {
    constexpr int NP = ClosedPairs<Q>::N;
    __shared__ __align__(16) ClosedPair tab[2 * NP];
    const long long row = (long long)(g.nx + 2) * Q, plane = row * (g.ny + 2);
    if (threadIdx.x < 2 * NP) {
        const int side = threadIdx.x >= NP, q = threadIdx.x - side * NP;
        const FacePairs& fp = side ? hi : lo;
        const int l = fp.l[q];
        // the plane next to the ghost, shifted by -c in the tangential directions
        const int in = side ? -1 : 1;
        const int dx = axis == 0 ? in : -fp.cx[q], dy = axis == 1 ? in : -fp.cy[q], dz = axis == 2 ? in : -fp.cz[q];
        tab[threadIdx.x] = ClosedPair{(long long)dx * Q + dy * row + dz * plane + l, l, fp.m[q], fp.cy[q], 0};
    }
    __syncthreads();
    const int e = blockIdx.x * 128 + threadIdx.x;
    const int a = e / NP + 1, b = blockIdx.y + 1;           // tangential indices
    const ClosedPair t0 = tab[e - (a - 1) * NP], t1 = tab[NP + e - (a - 1) * NP];
    if (a > (axis == 0 ? g.ny : g.nx)) return;
    const int j = axis == 0 ? a : axis == 1 ? 0 : b;
    const long long o0 = (axis == 0 ? 0 : a) * (long long)Q + j * row + (axis == 2 ? 0 : b) * plane;
    const long long o1 = o0 + (axis == 0 ? (g.nx + 1) * (long long)Q : axis == 1 ? (g.ny + 1) * row : (g.nz + 1) * plane);
    auto wrapped = [&](int js) { return wrap ? (js == 0 ? g.ny * row : (js == g.ny + 1 ? -g.ny * row : 0LL)) : 0LL; };
    const R r0 = f2[o0 + t0.l], r1 = f2[o1 + t1.l];
    const R p0 = f1[o0 + t0.d + wrapped(j - t0.cy)], p1 = f1[o1 + t1.d + wrapped(j - t1.cy)];
    f1[o0 + t0.m] = r0;
    f1[o0 + t0.l] = p0;
    f1[o1 + t1.m] = r1;
    f1[o1 + t1.l] = p1;
}

// inflow at i = 0 and zero-gradient outflow at i = nx+1: k_inflow of boundary.cuh with a
// thread per (direction, j); grid y over k
template <int Q, typename R>
__global__ void __launch_bounds__(256) k_ref_inflow(R* __restrict__ f, const R* __restrict__ uvel, R rho0, R cosd, R sind, RefGrid g) {
    __shared__ R tw[Q], tx[Q], ty[Q];
    __shared__ int ts[Q];
    if (threadIdx.x < Q) {
        const int l = threadIdx.x;
        const int s = lat_cx(l) > 0 ? lat_opposite(l) : l;   // the direction whose corrected value goes to ghost l
        ts[l] = s;
        tw[l] = lat_w<Q, R>(s);
        tx[l] = (R)lat_cx(s);
        ty[l] = (R)lat_cy(s);
    }
    __syncthreads();
    const int e = blockIdx.x * 256 + threadIdx.x;
    const int j = e / Q + 1, l = e - (j - 1) * Q, k = blockIdx.y + 1;
    if (j > g.ny) return;
    R* row = f + g.cell(0, j, k) * Q;
    const R uu = uvel[k - 1];
    const R cs2 = R(1) / R(3);
    const R in = row[Q + ts[l]] - R(2) * tw[l] * rho0 * (tx[l] * uu * cosd + ty[l] * uu * sind) / cs2;
    const R out = row[(long long)g.nx * Q + l];
    row[l] = in;
    row[(long long)(g.nx + 1) * Q + l] = out;
}

// forcings_apply: f += feq2(rho, u - F/rho) - feq2(rho, u) at interior cells with
// rho > 0 (m_forcings_apply_kernel.F90:47-213; second-order equilibria), in the
// closed form w rho [3 dcu + 4.5 dcu (2 cu + dcu) - 1.5 (2 u.du + du.du)].
template <int Q, typename R = float>
__global__ void __launch_bounds__(128) k_ref_forcings_apply(R* f, const R* force, const R* rho,
                                                            const R* u, const R* v, const R* w, RefGrid g) {
    __shared__ R sm[128 * Q];
    const int i0 = blockIdx.x * 128 + 1, j = blockIdx.y + 1, k = blockIdx.z + 1;
    const int n = min(128, g.nx + 1 - i0);
    const int t = threadIdx.x;
    if (n <= 0) return;
    tile_load<Q>(sm, f, g.cell(i0, j, k), n);
    __syncthreads();
    if (t < n) {
        const long long c = g.cell(i0 + t, j, k);
        const R rr = rho[c];
        if (rr > R(0.0)) {
            const R ux = u[c], uy = v[c], uz = w[c];
            const R dux = -force[3 * c] / rr, duy = -force[3 * c + 1] / rr, duz = -force[3 * c + 2] / rr;
            const R dusq = dux * (R(2.0) * ux + dux) + duy * (R(2.0) * uy + duy) + duz * (R(2.0) * uz + duz);
            R* p = sm + t * Q;
            p[0] += lat_w<Q, R>(0) * rr * (-R(1.5) * dusq);
#pragma unroll
            for (int l = 1; l < Q; l += 2) {
                const int cx = lat_cx(l), cy = lat_cy(l), cz = lat_cz(l);
                const R cu = cdot(cx, cy, cz, ux, uy, uz);
                const R dcu = cdot(cx, cy, cz, dux, duy, duz);
                const R wr = lat_w<Q, R>(l) * rr;
                const R dE = wr * (R(4.5) * dcu * (R(2.0) * cu + dcu) - R(1.5) * dusq);
                const R dO = wr * R(3.0) * dcu;
                p[l] += dE + dO;
                p[l + 1] += dE - dO;
            }
        }
    }
    __syncthreads();
    tile_store<Q>(sm, f, g.cell(i0, j, k), n);
}

// inflow_turbulence_forcing: df(l,j,k) = feq(rho,u+ampl*uu) - feq(rho,u) at i = iturb
// (m_inflow_turbulence_forcing.F90:44-128), evaluated as a difference of offsets
template <int Q, typename R = float>
__global__ void k_ref_turb_forcing(R* df, const R* rho, const R* u, const R* v, const R* w,
                                   const R* uu, const R* vv, const R* ww, R ampl, int lit, int ip,
                                   int ibgk, RefGrid g) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
    if (j > g.ny) return;
    const long long c = g.cell(ip, j, k);
    const long long t = (long long)(j - 1) + (long long)g.ny * ((long long)(k - 1) + (long long)g.nz * lit);
    const R r = rho[c];
    const R ux = u[c], uy = v[c], uz = w[c];
    const R dux = ampl * uu[t], duy = ampl * vv[t], duz = ampl * ww[t];
    const bool cubic = ibgk == 3;
    const R usq = ux * ux + uy * uy + uz * uz;
    const R dusq = dux * (R(2.0) * ux + dux) + duy * (R(2.0) * uy + duy) + duz * (R(2.0) * uz + duz);
    const R usq2 = usq + dusq;
    R* o = df + ((long long)(j - 1) + (long long)g.ny * (k - 1)) * Q;
    o[0] = lat_w<Q, R>(0) * r * (-R(1.5) * dusq);
#pragma unroll
    for (int l = 1; l < Q; l += 2) {
        const int cx = lat_cx(l), cy = lat_cy(l), cz = lat_cz(l);
        const R wr = lat_w<Q, R>(l) * r;
        const R cu = cdot(cx, cy, cz, ux, uy, uz);
        const R dcu = cdot(cx, cy, cz, dux, duy, duz);
        const R cun = cu + dcu;
        const R E = wr * (R(4.5) * dcu * (R(2.0) * cu + dcu) - R(1.5) * dusq);
        R od = R(3.0) * dcu;
        if (cubic) od += R(4.5) * dcu * (cun * cun + cun * cu + cu * cu - usq2) - R(4.5) * cu * dusq;
        const R O = wr * od;
        o[l] = E + O;
        o[l + 1] = E - O;
    }
}

// inflow_turbulence_apply: f(l,ip,j,k) += df(l,j,k) (m_inflow_turbulence_apply.F90:19-28)
template <typename R = float>
__global__ void k_ref_turb_apply(R* f, const R* df, int ip, RefGrid g) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;   // over (l, j)
    const int k = blockIdx.y + 1;
    const int nl = g.nl;
    if (e >= nl * g.ny) return;
    const int l = e % nl, j = e / nl + 1;
    f[g.cell(ip, j, k) * nl + l] += df[((long long)(j - 1) + (long long)g.ny * (k - 1)) * nl + l];
}

// fillghosts: ghost cells copy the nearest interior cell (m_fillghosts.F90:18-29)
template <typename R = float>
__global__ void k_ref_fillghosts(R* f, RefGrid g) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
    if (i > g.nx + 1) return;
    const int i1 = min(max(i, 1), g.nx), j1 = min(max(j, 1), g.ny), k1 = min(max(k, 1), g.nz);
    if (i1 == i && j1 == j && k1 == k) return;
    const int nl = g.nl;
    const R* s = f + g.cell(i1, j1, k1) * nl;
    R* d = f + g.cell(i, j, k) * nl;
    for (int l = 0; l < nl; ++l) d[l] = s[l];
}

}  // namespace lbm
