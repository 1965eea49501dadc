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

}  // namespace lbm
