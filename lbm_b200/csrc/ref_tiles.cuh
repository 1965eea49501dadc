// ref_tiles.cuh -- moving pieces of a reference-layout array
// f(nl,0:nx+1,0:ny+1,0:nz+1) (l fastest) between global and shared memory in
// 16-byte words.
//
// A run of cells is contiguous, but with nl = 19 or 27 it starts on any
// element, so neither the run nor its rows are 16-byte aligned.  Everything
// here therefore keeps a run in shared memory at the offset its address has
// within a 16-byte word (its phase): whole words of the run are whole words
// there too and move as such; the words at its two ends move element by
// element.  Nothing outside the run is read or written.  The copies to shared
// memory are cp.async, so a thread puts all its words in flight at once.
#pragma once

#include "common.cuh"

namespace lbm {

__device__ __forceinline__ void cp_async16(void* sm, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(sm)), "l"(g) : "memory");
}
template <typename R>
__device__ __forceinline__ void cp_async_elem(R* sm, const R* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(sm)), "l"(g),
                 "n"((int)sizeof(R)) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// elements of a 16-byte word, and the phase of an address in elements
template <typename R>
__host__ __device__ constexpr int word_elems() { return 16 / (int)sizeof(R); }
template <typename R>
__host__ __device__ __forceinline__ int phase_of(const R* p) {
    return (int)((reinterpret_cast<uintptr_t>(p) / sizeof(R)) % word_elems<R>());
}

// word w of the run of n elements at g to shared memory: sm is word aligned and
// holds element e of the run at sm[ph + e], ph the phase of g.  Words are
// counted from the one that holds element 0.
template <typename R>
__device__ __forceinline__ void run_load_word(R* sm, const R* g, int ph, int n, int w) {
    constexpr int V = word_elems<R>();
    const int e = w * V - ph;            // first element of the word, in the run if 0 <= e
    if (e >= 0 && e + V <= n) {
        cp_async16(sm + ph + e, g + e);
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (e + v >= 0 && e + v < n) cp_async_elem(sm + ph + e + v, g + e + v);
    }
}

// ---- tiles of T consecutive cells -------------------------------------------------
//
// The cell-wise kernels walk an array in tiles of T consecutive cells, a
// thread per cell, in blocks that stay on their SM and fetch the next tile (and
// its scalars) while they work on the current one.  Tiles run through the rows
// j = 1..ny of a plane without regard to row ends (ALL: through the whole
// array), so short rows leave no thread idle; the i ghosts they pass over are
// read and never written.
template <int Q, typename R, int T>
struct CellTile {
    static constexpr int V = word_elems<R>();
    static constexpr int WORDS = (T * Q + 2 * (V - 1)) / V;   // words a tile may touch
    static constexpr int BUF = (WORDS + 1) * V;                    // elements of a tile buffer
};

// tile t of the interior rows (k = 1..nz, tiles per plane tp) or of all cells
struct TileAt {
    long long c0;      // first cell
    int n;             // cells
    int k;             // plane (interior tiles)
    unsigned q0;       // first cell's index in the plane's rows j = 1..ny (interior tiles)
};
template <bool ALL, int T>
__device__ __forceinline__ TileAt tile_at(const RefGrid& g, unsigned t, unsigned tp) {
    TileAt a;
    if (ALL) {
        a.c0 = (long long)t * T;
        a.n = (int)min((long long)T, g.ncell() - a.c0);
        a.k = 0;
        a.q0 = 0;
    } else {
        const unsigned per_plane = (unsigned)(g.nx + 2) * (unsigned)g.ny, k = t / tp;
        a.q0 = (t - k * tp) * T;
        a.k = (int)k + 1;
        a.n = (int)min((unsigned)T, per_plane - a.q0);
        a.c0 = g.cell(0, 1, a.k) + a.q0;
    }
    return a;
}
// tiles of a plane's interior rows, and of the whole array
inline unsigned plane_tiles(const RefGrid& g, int T) { return ((unsigned)(g.nx + 2) * (unsigned)g.ny + T - 1) / T; }
inline unsigned all_tiles(const RefGrid& g, int T) { return (unsigned)((g.ncell() + T - 1) / T); }

// the n cells from c0 on to a tile buffer; their first element lands at phase_of(f + c0 Q)
template <int Q, int T, typename R>
__device__ __forceinline__ void tile_fetch(R* sm, const R* f, long long c0, int n) {
    const R* g = f + c0 * Q;
    const int ph = phase_of(g);
    for (int w = threadIdx.x; w < CellTile<Q, R, T>::WORDS; w += T) run_load_word(sm, g, ph, n * Q, w);
}

// a tile buffer back to the cells whose bit in `cells` (T / 32 words of shared
// memory) is set; whole: all of them are
template <int Q, int T, typename R>
__device__ __forceinline__ void tile_put(const R* sm, R* f, long long c0, int n, const unsigned* cells, bool whole) {
    constexpr int V = word_elems<R>();
    R* g = f + c0 * Q;
    const int ph = phase_of(g), m = n * Q;
    auto on = [&](int e) { const int c = e / Q; return (cells[c >> 5] >> (c & 31)) & 1u; };
    for (int w = threadIdx.x; w < CellTile<Q, R, T>::WORDS; w += T) {
        const int e = w * V - ph;
        if (e >= 0 && e + V <= m && (whole || (on(e) && on(e + V - 1)))) {
            *reinterpret_cast<uint4*>(g + e) = *reinterpret_cast<const uint4*>(sm + ph + e);
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v)
                if (e + v >= 0 && e + v < m && (whole || on(e + v))) g[e + v] = sm[ph + e + v];
        }
    }
}

}  // namespace lbm
