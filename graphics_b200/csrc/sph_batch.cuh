// sph_batch.cuh -- a batch's per-scene reductions over chunks of its scenes'
// ranges, and the loop decisions that sweep B's leading blocks make with them.
#pragma once
#include "sph_kernels.cuh"

// an upper bound on the chunks of all scenes: sum ceil(n_s / C) <= n / C + scenes
inline int batch_chunks(int n_cap, int nscenes) { return n_cap / BATCH_CHUNK + nscenes + 1; }

__device__ __forceinline__ void scene_range(const DevScene& s, int sc, int& a, int& b) {
    const GridGeom& G = s.b.geom[sc];
    a = s.cell_start[G.key0];
    b = s.cell_start[G.key1];
}

// the scene of chunk `bid` (chunk0 ascending; empty scenes have no chunks)
__device__ __forceinline__ int chunk_scene(const DevScene& s, int nscenes, int bid) {
    int lo = 0, hi = nscenes - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s.b.chunk0[mid] <= bid) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Density loop (DIV 0: mean rho_adv, aux0) or divergence loop (1: mean
// Drho/Dt, aux1): block bid of nblocks (batch_chunks) takes the chunk of that
// number, if its scene is active.  Same rules as the single-scene decision
// (DFSPH.cpp:566-700, 740-1024 with the FP64 mean and caps).  It needs sweep
// A's results only, so it runs beside the sweep B of the same iteration, which
// reads active_b: as a kernel after it, it took 8 us of an iteration's 79 at
// 12 scenes of 5 000 to 60 000 particles.
template <int BS, int DIV>
__device__ __forceinline__ void batch_decide(const DevScene& s, const SolverConst& c, int bid, int nblocks,
                                             double goal_abs, double goal_rel, int min_it, int max_it,
                                             cudaGraphConditionalHandle h, int use_handle) {
    const int nscenes = s.nscenes;
    __shared__ double sh[BS / 32];
    __shared__ bool last;
    const int total = s.b.chunk0[nscenes];
    const int sc = bid < total ? chunk_scene(s, nscenes, bid) : -1;
    if (sc >= 0 && s.b.active_b[sc]) {  // uniform over the block
        int a, b;
        scene_range(s, sc, a, b);
        const int k = bid - s.b.chunk0[sc];
        const int c0 = a + k * BATCH_CHUNK, c1 = min(b, c0 + BATCH_CHUNK);
        const float* v = DIV ? s.aux1 : s.aux0;
        double acc = 0.0;
        constexpr int LD = 16;  // loads in flight together
        for (int i0 = c0 + (int)threadIdx.x; i0 < c1; i0 += LD * BS) {
            float x[LD];
#pragma unroll
            for (int q = 0; q < LD; ++q) x[q] = i0 + q * BS < c1 ? v[i0 + q * BS] : 0.f;
#pragma unroll
            for (int q = 0; q < LD; ++q) acc += (double)x[q];
        }
        const double part = block_sum_double<BS>(acc, sh);
        if (threadIdx.x == 0) {
            s.partial[bid] = part;
            __threadfence();
            const int nch = s.b.chunk0[sc + 1] - s.b.chunk0[sc];
            last = atomicAdd(&s.b.sticket[sc], 1u) == (unsigned)(nch - 1);
        }
        __syncthreads();
        if (last) {
            // the scene's last chunk: its chunks' sums in chunk order, loaded
            // by all threads (one thread alone waits out the L2 latency per
            // chunk)
            __shared__ double part_of[BS];
            double tot = 0.0;
            __threadfence();
            const int q0 = s.b.chunk0[sc], q1 = s.b.chunk0[sc + 1];
            for (int q = q0; q < q1; q += BS) {
                if (q + (int)threadIdx.x < q1) part_of[threadIdx.x] = __ldcg(s.partial + q + threadIdx.x);
                __syncthreads();
                if (threadIdx.x == 0)
                    for (int i = 0; i < min(BS, q1 - q); ++i) tot += part_of[i];
                __syncthreads();
            }
            if (threadIdx.x == 0) {
                s.b.sticket[sc] = 0u;
                const double n = (double)(b - a);
                bool crit;
                int cont;
                if (!DIV) {
                    const int it = ++s.b.it_density[sc];
                    ++s.b.total_it_density[sc];
                    const double err = (tot / n - (double)c.rho0) / (double)c.rho0;
                    s.b.err_density[sc] = err;
                    crit = err > goal_rel;
                    cont = (crit || it < min_it) && it < max_it;
                    if (!cont && crit) s.b.status[sc] |= 1u;
                    if (!(err == err)) { cont = 0; s.b.status[sc] |= 4u; }
                } else {
                    const int it = ++s.b.it_div[sc];
                    ++s.b.total_it_div[sc];
                    const double avg = tot / n;
                    s.b.err_div[sc] = avg;
                    const double dtd = (double)s.b.dt[sc];
                    crit = goal_abs > 0 ? (avg > goal_abs) : (avg * dtd / (double)c.rho0 > goal_rel);
                    cont = (crit || it < min_it) && it <= max_it;
                    if (!cont && crit) s.b.status[sc] |= 2u;
                    if (!(avg == avg)) { cont = 0; s.b.status[sc] |= 4u; }
                }
                if (!cont) s.b.active[sc] = 0;
            }
        }
        __syncthreads();
    }
    // the last block to finish decides whether the loop runs again
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&s.st->ticket[0], 1u) == (unsigned)(nblocks - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int any = 0;
    unsigned st_or = 0u;
    for (int i = threadIdx.x; i < nscenes; i += BS) {
        any |= ((volatile int*)s.b.active)[i];
        st_or |= ((volatile unsigned*)s.b.status)[i];
    }
    any = __syncthreads_or(any);
    __shared__ unsigned sst;
    if (threadIdx.x == 0) sst = 0u;
    __syncthreads();
    if (st_or) atomicOr(&sst, st_or);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (DIV) ++s.st->it_div;
        else ++s.st->it_density;
        s.st->status |= sst;
        s.st->cont = any;
        s.st->ticket[0] = 0u;
        if (use_handle) cudaGraphSetConditional(h, any ? 1u : 0u);
    }
}
