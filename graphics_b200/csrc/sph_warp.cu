// sph_warp.cu -- neighbour lists, a warp for a few consecutive particles.
//
// A thread per particle walks some 220 candidates and 30 neighbours one
// after the other: a small scene has too few warps on the chip to hide that
// (1 k particles: 44 to 53 us, by mode), and a large one spends its issue slots
// on the loop and on the lanes that wait for the longest walk.  Here a warp
// takes up to 16 consecutive sorted particles, cell by cell: the candidates of a
// cell (its 27 cells' records, in the reference's order) go into the lanes'
// registers once, each particle of the cell tests 32 of them per
// instruction, and a ballot gives every hit its place in the list.  Then the
// lanes take one list entry each for the terms; the sums run in list order,
// one lane per sum (WCSPH's density: per block of it), so every result is the
// one k_build (sph_grid.cu) gives, bit for bit: the same cells in the same
// order, the same float cut test, the same cap.
#include <algorithm>

#include "sph_build.cuh"

namespace {
constexpr int GROUP = 16;        // particles per warp at most
constexpr int ROUNDS = 8;        // candidates per window: 32 a round
constexpr int WINDOW = 32 * ROUNDS;
constexpr int LIST = 52;         // list entries kept in shared memory (cap <= 48), whole 16-byte groups
constexpr int SUMS = 8;          // lanes per particle in the sums
constexpr int TROW = 33;         // stride of a sum's 32 factors: the lanes of the sums read distinct banks

template <int MODE>
struct WarpSmem {
    static constexpr int N = MODE ? BuildSums<MODE ? MODE : 1>::N : 1;
    static constexpr int PAIR = MODE ? 2 : 0;  // particles whose sums run together
    alignas(16) int list[GROUP * LIST];        // read as int4
    union {
        int cand[WINDOW];
        float uv[(PAIR ? PAIR : 1) * 2 * N * TROW];
    };
    float sum[GROUP * SUMS];
};
static_assert(LIST % 4 == 0 && sizeof(WarpSmem<0>) % 16 == 0 && sizeof(WarpSmem<3>) % 16 == 0,
              "every particle's row of every warp's list on 16 bytes");

// One block size: its warps share nothing but the statistics, and 64 or 256
// threads are no faster (event-timed 64 / 128 / 256: 1 k particles 12.7 / 12.7 /
// 12.7 us, 8 k 19.1 / 18.9 / 20.8, 27 k 36 / 36 / 40, 46 k 49 / 49 / 53, 64 k
// 78 / 78 / 83), while every instantiation makes the module longer that a
// process loads for its first small scene.
constexpr int NT = 128;

template <int MODE>
__global__ void __launch_bounds__(NT) k_warp_build(const __grid_constant__ DevScene s, const __grid_constant__ GridGeom g,
                                                   const __grid_constant__ SolverConst c, int group) {
    constexpr int WPB = NT / 32;
    using Smem = WarpSmem<MODE>;
    extern __shared__ int4 warp_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    Smem& m = reinterpret_cast<Smem*>(warp_smem)[wid];
    const unsigned below = (1u << lane) - 1u;
    const int n = s.st->n_active;
    int ntot = 0, over = 0, nmax = 0;
    double dsum = 0.0;  // MODE 4: the particles' Drho/Dt
    for (int p0 = (blockIdx.x * WPB + wid) * group; p0 < n; p0 += gridDim.x * WPB * group) {
        const int ng = min(group, n - p0);
        // lane l < ng: particle p0 + l
        float4 pa = make_float4(0.f, 0.f, 0.f, 0.f);
        int cx = 0, cy = 0, cz = 0, key = -1, cnt = 0;
        if (lane < ng) {
            pa = s.pos[p0 + lane];
            const GridGeom& G = s.nscenes > 1 ? s.b.geom[scene_of(pa)] : g;
            cx = cell_coord(pa.x, G.min[0], G.divisor);
            cy = cell_coord(pa.y, G.min[1], G.divisor);
            cz = cell_coord(pa.z, G.min[2], G.divisor);
            key = cell_key(G, cx, cy, cz);
        }
        for (unsigned todo = (1u << ng) - 1u; todo;) {
            // the particles of one cell
            const int l0 = __ffs(todo) - 1;
            const unsigned same = __ballot_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, l0)) & todo;
            todo &= ~same;
            // lane l < 27: cell l of the scan, its records and its place
            // among the candidates
            int2 s0 = make_int2(0, 0), s1 = s0;
            {
                const int x0 = __shfl_sync(0xffffffffu, cx, l0), y0 = __shfl_sync(0xffffffffu, cy, l0),
                          z0 = __shfl_sync(0xffffffffu, cz, l0);
                const int sc = s.nscenes > 1 ? scene_of(make_float4(0.f, 0.f, 0.f, __shfl_sync(0xffffffffu, pa.w, l0))) : 0;
                const GridGeom& G = s.nscenes > 1 ? s.b.geom[sc] : g;
                const int x = x0 + lane % 3 - 1, y = y0 + lane / 3 % 3 - 1, z = z0 + lane / 9 - 1;
                if (lane < 27 && cell_inside(G, x, y, z)) {
                    const int k = cell_key(G, x, y, z);
                    s0 = __ldg(s.cstart2 + k);
                    s1 = __ldg(s.cstart2 + k + 1);
                }
            }
            const int nf = s1.x - s0.x, num = nf + (s1.y - s0.y);
            int at = num;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, at, o);
                if (lane >= o) at += t;
            }
            const int total = __shfl_sync(0xffffffffu, at, 31);
            at -= num;
            for (int w0 = 0; w0 < total; w0 += WINDOW) {
                __syncwarp();
                for (int k = max(0, w0 - at); k < num && at + k < w0 + WINDOW; ++k)
                    m.cand[at + k - w0] = k < nf ? s0.x + k : (int)((unsigned)(s0.y + k - nf) | BND_FLAG);
                __syncwarp();
                const int here = min(WINDOW, total - w0);
                int e[ROUNDS];
                float qx[ROUNDS], qy[ROUNDS], qz[ROUNDS];
#pragma unroll
                for (int r = 0; r < ROUNDS; ++r) {
                    // none: a position beyond any cut
                    e[r] = 0;
                    qx[r] = qy[r] = qz[r] = 1e18f;
                    if (32 * r + lane < here) {
                        e[r] = m.cand[32 * r + lane];
                        const float4 q = __ldg((e[r] < 0 ? s.bpos : s.pos) + (e[r] & (int)BND_MASK));
                        qx[r] = q.x;
                        qy[r] = q.y;
                        qz[r] = q.z;
                    }
                }
                for (unsigned left = same; left; left &= left - 1u) {
                    const int j = __ffs(left) - 1;
                    const float px = __shfl_sync(0xffffffffu, pa.x, j), py = __shfl_sync(0xffffffffu, pa.y, j),
                                pz = __shfl_sync(0xffffffffu, pa.z, j);
                    int kj = __shfl_sync(0xffffffffu, cnt, j);  // hits so far, the first `cap` are kept
                    int* const row = m.list + j * LIST;
#pragma unroll
                    for (int r = 0; r < ROUNDS; ++r) {
                        if (32 * r >= here) break;
                        const bool hit = dis_square_rn(px, py, pz, qx[r], qy[r], qz[r]) < c.h2cut && e[r] != p0 + j;
                        const unsigned hits = __ballot_sync(0xffffffffu, hit);
                        const int k = kj + __popc(hits & below);
                        if (hit && k < c.cap) row[k] = e[r];
                        kj += __popc(hits);
                    }
                    if (lane == j) cnt = kj;
                }
            }
        }
        __syncwarp();
        const int kept = min(cnt, c.cap);
        if (lane < ng) {
            s.ncount[p0 + lane] = kept;
            over += cnt - kept;
            ntot += kept;
            nmax = max(nmax, kept);
        }
        // the lists, 16 bytes of a particle's per lane (entries past the
        // count are never read: every sweep masks them)
        const int most = __reduce_max_sync(0xffffffffu, kept);
        {
            const int j = lane & (GROUP - 1);
            const int kj = __shfl_sync(0xffffffffu, kept, j);
            for (int gi = lane / GROUP; 4 * gi < most; gi += 32 / GROUP)
                if (4 * gi < kj)
                    reinterpret_cast<int4*>(s.nbr)[(size_t)gi * c.stride + p0 + j] =
                        *reinterpret_cast<const int4*>(m.list + j * LIST + 4 * gi);
        }
        if (MODE != 0) {
            constexpr int M = MODE ? MODE : 1;
            constexpr int N = Smem::N, PAIR = MODE ? Smem::PAIR : 1;
            constexpr int R = MODE == 2 ? (LIST - 4) / DENS_BLOCK : N;  // results per particle (cap <= LIST - 4)
            float4 va = make_float4(0.f, 0.f, 0.f, 0.f);
            if (build_has_div(MODE) && lane < ng) va = s.pv[2 * (p0 + lane) + 1];
            for (int j0 = 0; j0 < ng; j0 += PAIR) {
                // lane b * SUMS + i: sum i (MODE 2: block i of the one sum) of particle j0 + b
                const int b = lane / SUMS, i = lane % SUMS;
                const bool sums = b < PAIR && i < R && j0 + b < ng;
                float acc = 0.f;
                if (MODE != 2) {
                    BuildSums<M> a;
                    sums_begin<M>(c, make_float4(0.f, 0.f, 0.f, __shfl_sync(0xffffffffu, pa.w, (j0 + b) & 31)), a);
#pragma unroll
                    for (int q = 0; q < N; ++q)
                        if (i == q) acc = a.v[q];
                }
                const int mykept = __shfl_sync(0xffffffffu, kept, (j0 + b) & 31);
                int kmax = 0;
#pragma unroll
                for (int t = 0; t < PAIR; ++t) kmax = max(kmax, __shfl_sync(0xffffffffu, kept, (j0 + t) & 31));
                for (int k0 = 0; k0 < kmax; k0 += 32) {
#pragma unroll
                    for (int t = 0; t < PAIR; ++t) {
                        const int j = (j0 + t) & 31;
                        const float4 pj = make_float4(__shfl_sync(0xffffffffu, pa.x, j), __shfl_sync(0xffffffffu, pa.y, j),
                                                      __shfl_sync(0xffffffffu, pa.z, j), __shfl_sync(0xffffffffu, pa.w, j));
                        float4 vj = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (build_has_div(MODE)) {
                            vj.x = __shfl_sync(0xffffffffu, va.x, j);
                            vj.y = __shfl_sync(0xffffffffu, va.y, j);
                            vj.z = __shfl_sync(0xffffffffu, va.z, j);
                        }
                        if (k0 + lane < __shfl_sync(0xffffffffu, kept, j)) {
                            const unsigned e = (unsigned)m.list[j * LIST + k0 + lane];
                            const bool bnd = (e & BND_FLAG) != 0u;
                            float4 pb, vb = make_float4(0.f, 0.f, 0.f, 0.f);
                            // pv / bpv hold {the position (boundary: with
                            // its volume) of pos / bpos, the velocity}
                            if (build_has_div(MODE)) ld_record32((bnd ? s.bpv : s.pv) + 2 * (size_t)(e & BND_MASK), pb, vb);
                            else pb = __ldg((bnd ? s.bpos : s.pos) + (e & BND_MASK));
                            BuildSums<M> u, v;
                            pair_terms<M>(c, pj, vj, bnd, pb, vb, u, v);
#pragma unroll
                            for (int q = 0; q < N; ++q) {
                                m.uv[(2 * (t * N + q)) * TROW + lane] = u.v[q];
                                m.uv[(2 * (t * N + q) + 1) * TROW + lane] = v.v[q];
                            }
                        }
                    }
                    __syncwarp();
                    if (sums) {
                        // MODE 2: block i is DENS_BLOCK of these 32 entries or none
                        const int first = MODE == 2 ? i * DENS_BLOCK - k0 : 0;
                        const int end = min(MODE == 2 ? min(32, first + DENS_BLOCK) : 32, mykept - k0);
                        const float* const U = m.uv + 2 * (b * N + (MODE == 2 ? 0 : i)) * TROW;
                        if (first >= 0)
#pragma unroll 4
                            for (int k = first; k < end; ++k) acc = fmaf(U[k], U[TROW + k], acc);
                    }
                    __syncwarp();
                }
                if (sums) m.sum[(j0 + b) * SUMS + i] = acc;
            }
            __syncwarp();
            if (lane < ng) {
                BuildSums<M> a;
                if (MODE == 2) sums_begin<M>(c, pa, a);
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    if (MODE == 2) a.v[0] += m.sum[lane * SUMS + q];
                    else a.v[q] = m.sum[lane * SUMS + q];
                }
                const double dd = sums_finish<M>(s, c, p0 + lane, pa, a);
                if (MODE == 4) dsum += dd;
            }
            __syncwarp();
        }
    }
    __shared__ int sh[WPB];
    const int tot = block_sum_int<NT>(ntot, sh);
    const int ov = block_sum_int<NT>(over, sh);
    const int mx = block_max_int<NT>(nmax, sh);
    if (threadIdx.x == 0) {
        if (tot) atomicAdd(&s.st->nbr_total, (unsigned long long)tot);
        if (ov) { atomicAdd(&s.st->overflow, ov); atomicOr(&s.st->status, 8u); }
        if (mx) atomicMax(&s.st->max_nbrs, mx);
    }
    if (MODE == 4) {
        // the block's part of the iteration's FP64 sum of Drho/Dt (as
        // k_df_div_a; a batch, mode 5, reduces per scene in batch_decide)
        __shared__ double shd[WPB];
        const double bsum = block_sum_double<NT>(dsum, shd);
        if (threadIdx.x == 0) s.partial[blockIdx.x] = bsum;
    }
}
}  // namespace

// particles per warp: enough warps for every SM first
static int warp_group(int n_max) { return std::min(GROUP, std::max(1, n_max / (148 * 16))); }
int warp_build_blocks(int n_max) {
    const int per = NT / 32 * warp_group(n_max), n = n_max > 0 ? n_max : 1;
    return (n + per - 1) / per;
}

void launch_warp_build(const DevScene& s, const GridGeom& g, const SolverConst& c, int mode, int n_max, cudaStream_t st) {
    if (mode == 4 && s.nscenes > 1) mode = 5;
    const int group = warp_group(n_max), nb = warp_build_blocks(n_max);
#define ONE(M) case M: k_warp_build<M><<<nb, NT, sizeof(WarpSmem<M>) * (NT / 32), st>>>(s, g, c, group); break;
    switch (mode) { ONE(0) ONE(1) ONE(2) ONE(3) ONE(4) ONE(5) }
#undef ONE
}
