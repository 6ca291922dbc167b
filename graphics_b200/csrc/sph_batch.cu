// sph_batch.cu -- many independent DFSPH scenes in one set of arrays.
//
// A batch packs every scene's particles into the same sorted arrays: each
// scene has its own grid (its own box), and the scenes' cell keys occupy
// disjoint ranges [key0, key1) of one key space, so one counting sort per
// step sorts all scenes at once, every scene's particles end up contiguous,
// and no neighbour list crosses scenes.  The sweep kernels are the
// single-scene ones (they read the scene index from pos.w for the scene's
// grid and time step); what is per scene lives here:
//   * the CFL step (FP64 max |v| over the scene's range),
//   * the loop decisions: the FP64 mean of rho_adv (density loop) or of
//     Drho/Dt (divergence loop) over the scene's range, the scene's own
//     iteration count and goal; a scene that has converged stops iterating
//     (its particles are skipped by the sweeps) while the others continue,
//     and the loop (a conditional graph node) runs while any scene is active.
// Each reduction runs over the scenes' contiguous ranges in chunks of
// BATCH_CHUNK particles, one block per chunk (a scene of 200k particles is
// 49 blocks, not one): the chunk's block sums (or maxima) go to partial[],
// the scene's last chunk to finish combines its chunks in chunk order and
// makes the scene's decision, and the last block of all makes the loop's
// (batch_decide in sph_batch.cuh, run by the leading blocks of sweep B).
// Sums are in a fixed order, so results are run-to-run deterministic.
#include "sph_batch.cuh"

namespace {
constexpr int NT = 256;

__global__ void k_batch_call_begin(DevScene s, int nscenes) {
    const int sc = blockIdx.x * blockDim.x + threadIdx.x;
    if (sc >= nscenes) return;
    s.b.total_it_density[sc] = 0;
    s.b.total_it_div[sc] = 0;
    s.b.status[sc] = 0u;
}

// active particles per scene after a neighbour search, and the scenes'
// first chunks (one thread: a prefix over the scenes)
__global__ void k_batch_count(DevScene s, int nscenes) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    int c = 0;
    for (int sc = 0; sc < nscenes; ++sc) {
        int a, b;
        scene_range(s, sc, a, b);
        s.b.n[sc] = b - a;
        s.b.chunk0[sc] = c;
        c += (b - a + BATCH_CHUNK - 1) / BATCH_CHUNK;
    }
    s.b.chunk0[nscenes] = c;
}

// start of a density (which 0) or divergence (which 1) loop
__global__ void k_batch_loop_reset(DevScene s, int nscenes, int which) {
    const int sc = blockIdx.x * blockDim.x + threadIdx.x;
    if (sc < nscenes) {
        s.b.active[sc] = s.b.active_b[sc] = s.b.n[sc] > 0 ? 1 : 0;
        if (which == 0) s.b.it_density[sc] = 0;
        else s.b.it_div[sc] = 0;
    }
    if (sc == 0) s.st->cont = 1;
}

// per-scene CFL step: dt = clamp(cfl * d / max|v|, dt_min, dt_max), FP64
// max over the scene's chunks (the maximum is order-independent)
__global__ void __launch_bounds__(NT) k_batch_cfl(DevScene s, int nscenes, float cfl, float d, float dt_max,
                                                  float dt_min) {
    const int bid = blockIdx.x;
    const int total = s.b.chunk0[nscenes];
    if (bid == 0)  // scenes without particles (no chunks): dt_max
        for (int q = threadIdx.x; q < nscenes; q += NT)
            if (s.b.chunk0[q + 1] == s.b.chunk0[q]) {
                s.b.vmax[q] = 0.0;
                s.b.dt[q] = dt_max;
            }
    if (bid >= total) return;
    const int sc = chunk_scene(s, nscenes, bid);
    int a, b;
    scene_range(s, sc, a, b);
    const int k = bid - s.b.chunk0[sc];
    const int c0 = a + k * BATCH_CHUNK, c1 = min(b, c0 + BATCH_CHUNK);
    double m = 0.0;
#pragma unroll 8
    for (int i = c0 + threadIdx.x; i < c1; i += NT) {
        const float4 v = s.vel[i];
        const double x = v.x, y = v.y, z = v.z;
        m = fmax(m, sqrt(x * x + y * y + z * z));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    __shared__ double sh[NT / 32];
    __shared__ bool last;
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double bm = 0.0;
        for (int i = 0; i < NT / 32; ++i) bm = fmax(bm, sh[i]);
        s.partial[bid] = bm;
        __threadfence();
        const int nch = s.b.chunk0[sc + 1] - s.b.chunk0[sc];
        last = atomicAdd(&s.b.sticket[sc], 1u) == (unsigned)(nch - 1);
    }
    __syncthreads();
    if (!last) return;
    // the scene's last chunk: the chunks' maxima, loaded by all threads
    __threadfence();
    double vmax = 0.0;
    for (int q = s.b.chunk0[sc] + threadIdx.x; q < s.b.chunk0[sc + 1]; q += NT) vmax = fmax(vmax, __ldcg(s.partial + q));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_down_sync(0xffffffffu, vmax, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = vmax;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < NT / 32; ++i) vmax = fmax(vmax, sh[i]);
        s.b.sticket[sc] = 0u;
        double dt = vmax > 0 ? (double)cfl * (double)d / vmax : (double)dt_max;
        if (dt > dt_max) dt = dt_max;
        if (dt < dt_min) dt = dt_min;
        s.b.vmax[sc] = vmax;
        s.b.dt[sc] = (float)dt;
    }
}
}  // namespace

static inline int blocks_for(int n, int nt) { return (n + nt - 1) / nt; }

void launch_batch_call_begin(const DevScene& s, int nscenes, cudaStream_t st) {
    k_batch_call_begin<<<blocks_for(nscenes, 128), 128, 0, st>>>(s, nscenes);
}
void launch_batch_count(const DevScene& s, int nscenes, cudaStream_t st) {
    k_batch_count<<<1, 32, 0, st>>>(s, nscenes);
}
void launch_batch_loop_reset(const DevScene& s, int nscenes, int which, cudaStream_t st) {
    k_batch_loop_reset<<<blocks_for(nscenes, 128), 128, 0, st>>>(s, nscenes, which);
}
void launch_batch_cfl(const DevScene& s, int nscenes, int n_cap, float cfl, float d, float dt_max, float dt_min,
                      cudaStream_t st) {
    k_batch_cfl<<<batch_chunks(n_cap, nscenes), NT, 0, st>>>(s, nscenes, cfl, d, dt_max, dt_min);
}
