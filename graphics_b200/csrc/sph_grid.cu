// sph_grid.cu -- uniform-grid neighbour search on the GPU.
//
// Replaces SphBase::gridSetup + SphBase::neighbourSearch
// (SphBase.cpp:849-1089).  The reference inserts every particle at the head
// of a per-cell linked list (solids first, then fluids, each in index order)
// and walks the 27 surrounding cells (x fastest, then y, then z;
// SphBase.cpp:980-986) and each list in list order, keeping a neighbour j when
// its float squared distance is < (d_i + d_j)^2 and stopping at 48 entries.
// The list order is therefore: per cell, fluids in descending (phase, index),
// then solids in descending (solid, index).
//
// Here: one counting sort per step by cell key (atomic histogram, exclusive
// scan, scatter), then a within-cell rank step that orders each cell's
// particles by descending global index -- exactly the reference's list order
// -- while reordering the particle state into the new layout.  Boundary
// particles are sorted once into their own cell table.  The neighbour-list
// kernel then walks the 27 cells in the reference's offset order, the fluid
// range of a cell before its boundary range, so the stored lists (and which
// entries a 48-cap truncates) are the reference's.  The cut test uses
// round-to-nearest float ops in the reference's evaluation order, so the
// neighbour sets are bit-identical.
#include "sph_build.cuh"

namespace {
constexpr int NT = 256;

// The counters' kernels are here, in the module that every solver needs: in
// DFSPH's, a process's first WCSPH or IISph step loaded that one too (2.5 -> 1.1
// and 4.1 -> 2.8 ms).
__global__ void k_step_begin(DevScene s) { stats_step_begin(s.st); }

// per-call counters: status bits are OR-ed and removals / dropped pairs
// summed over all steps of one API call
__global__ void k_call_begin(DevScene s) {
    DevStats* st = s.st;
    st->removed = 0;
    st->overflow = 0;
    st->zero_dis = 0;
    st->status = 0u;
    st->total_it_density = 0;
    st->total_it_div = 0;
}

__global__ void __launch_bounds__(NT) k_hash(DevScene s, GridGeom g, int integrate) {
    const int n = s.st->n_active;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s.st->pad0 = n;  // staged count
        if (integrate & 8) stats_step_begin(s.st);
    }
    int i = blockIdx.x * NT + threadIdx.x;
    int removed = 0, nan = 0;
    if (i < n) {
        float4 p, v;
        if (integrate & 7) {
            // Second loop 2.4: velocity = vel_adv; position += velocity*dt
            // (DFSPH.cpp:705-715), in round-to-nearest float ops.
            p = s.pos[i];
            const float dt = dt_of(s, p);
            v = s.pv[2 * i + 1];  // v_adv of the density loop
            p.x = __fadd_rn(p.x, __fmul_rn(v.x, dt));
            p.y = __fadd_rn(p.y, __fmul_rn(v.y, dt));
            p.z = __fadd_rn(p.z, __fmul_rn(v.z, dt));
            v.w = 0.f;
            s.pos_s[i] = p;
            s.vel_s[i] = v;
            s.gid_s[i] = s.gid[i];
            if (integrate & 4) {
                // the learned warm start's history of this step (as k_ws_post):
                // the step's kappa sum with the applied prediction, and the
                // step's (predicted error, divergence term); the sum restarts
                const float2 w = s.wsbuf[i];
                s.hist_s[i] = make_float4(s.ksum[i] + s.kwarm[i], w.x, w.y, 0.f);
                s.ksum[i] = 0.f;
            } else {
                s.hist_s[i] = s.hist[i];
            }
            if (integrate & 2) s.cA_s[i] = s.cA[i];  // DFSPH vorticity state carried through the sort
        } else {
            p = s.pos_s[i];
        }
        // the particle's scene grid (the only grid unless this is a batch)
        const GridGeom G = s.nscenes > 1 ? s.b.geom[scene_of(p)] : g;
        // SphFluid::removeOutsideParts test (SphBase.cpp:34-44, Vec23.h:193-194)
        bool in = G.smin[0] <= p.x && G.smin[1] <= p.y && G.smin[2] <= p.z && p.x <= G.smax[0] &&
                  p.y <= G.smax[1] && p.z <= G.smax[2];
        int key = g.nkeys - 1;
        if (in) {
            int cx = cell_coord(p.x, G.min[0], G.divisor);
            int cy = cell_coord(p.y, G.min[1], G.divisor);
            int cz = cell_coord(p.z, G.min[2], G.divisor);
            if (cell_inside(G, cx, cy, cz)) key = cell_key(G, cx, cy, cz);
            else removed = 1;
        } else {
            removed = 1;
            if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) nan = 1;
        }
        s.key[i] = key;
        s.slot[i] = atomicAdd(&s.cell_count[key], 1);
    }
    if (__syncthreads_or(removed)) {
        if (removed) atomicOr(&s.st->status, 16u | (nan ? 4u : 0u));
    }
}

// Everything that needs the cell starts only: the particles' arrival slots,
// the interleaved {fluid start, boundary start} per cell key (one 8-byte load
// per cell bound in the list build), the number of active particles, and the
// counts back to zero for the next search.
__global__ void __launch_bounds__(NT) k_scatter(DevScene s, int nk) {
    const int n = s.st->pad0;
    const int i = blockIdx.x * NT + threadIdx.x;
    if (i < n) s.tmp[s.cell_start[s.key[i]] + s.slot[i]] = i;
    if (i <= nk) {
        s.cstart2[i] = make_int2(s.cell_start[i], s.bcell_start[i]);
        s.cell_count[i] = 0;
    }
    if (i == 0) {
        const int act = s.cell_start[nk - 1];  // the dead key's start
        s.st->removed += n - act;
        s.st->n_active = act;
    }
}

// Exclusive scan of n counts by one block: 4096 a round, the next round's
// loads issued before the current one is summed.
constexpr int SCAN_NT = 1024;
__global__ void __launch_bounds__(SCAN_NT) k_scan(const int* __restrict__ in, int* __restrict__ out, int n) {
    __shared__ int wsum[SCAN_NT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    auto load = [&](int i) {
        int4 v = make_int4(0, 0, 0, 0);
        if (i + 3 < n) {
            v = *reinterpret_cast<const int4*>(in + i);
        } else {
            if (i < n) v.x = in[i];
            if (i + 1 < n) v.y = in[i + 1];
            if (i + 2 < n) v.z = in[i + 2];
        }
        return v;
    };
    int carry = 0;
    int4 nxt = load(4 * threadIdx.x);
    for (int base = 0; base < n; base += 4 * SCAN_NT) {
        const int i = base + 4 * threadIdx.x;
        const int4 v = nxt;
        nxt = load(i + 4 * SCAN_NT);
        const int sum = v.x + v.y + v.z + v.w;
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        int w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        const int before = carry + (wid ? __shfl_sync(0xffffffffu, w, wid - 1) : 0) + incl - sum;
        carry += __shfl_sync(0xffffffffu, w, 31);
        __syncthreads();
        const int4 o4 = make_int4(before, before + v.x, before + v.x + v.y, before + v.x + v.y + v.z);
        if (i + 3 < n) {
            *reinterpret_cast<int4*>(out + i) = o4;
        } else {
            if (i < n) out[i] = o4.x;
            if (i + 1 < n) out[i + 1] = o4.y;
            if (i + 2 < n) out[i + 2] = o4.z;
        }
    }
}

// For sorted slot q: its particle i, its cell range [a, b); its final place is
// a + #{particles of the cell with larger global index}.
__global__ void __launch_bounds__(NT) k_rank_reorder(DevScene s, int dead_key, int carry) {
    const int n = s.st->pad0;
    int q = blockIdx.x * NT + threadIdx.x;
    if (q >= n) return;
    int i = s.tmp[q];
    int key = s.key[i];
    if (key == dead_key) return;
    int a = s.cell_start[key], b = s.cell_start[key + 1];
    int my = s.gid_s[i], cnt = 0;
    for (int r = a; r < b; ++r) cnt += s.gid_s[s.tmp[r]] > my;
    int p = a + cnt;
    const float4 x = s.pos_s[i], v = s.vel_s[i];
    s.pos[p] = x;
    s.vel[p] = v;
    s.pv[2 * p] = x;
    s.pv[2 * p + 1] = v;
    s.prv[2 * p + 1] = v;
    s.pk[p] = make_float4(x.x, x.y, x.z, 0.f);
    s.gid[p] = my;
    if (carry & 1) s.hist[p] = s.hist_s[i];
    if (carry & 2) s.cA[p] = s.cA_s[i];
    if (carry & 4) {
        const float4 b = s.cB_s[i];
        s.cB[p] = b;
        // the record of the PCISPH / IISPH_M non-pressure forces
        s.prv[2 * p] = x;
        s.prv[2 * p + 1] = make_float4(v.x, v.y, v.z, b.w);
    }
    if (carry & 8) s.cC[p] = s.cC_s[i];
}

// the interleaved starts again after the boundary alone was re-sorted
__global__ void k_merge_starts(DevScene s, int nk) {
    const int k = blockIdx.x * NT + threadIdx.x;
    if (k <= nk) s.cstart2[k] = make_int2(s.cell_start[k], s.bcell_start[k]);
}

// Ints per thread of the shared-memory list staging (>= the cap of 48, a
// multiple of 4 so that every row starts on a 16-byte boundary; 52 also
// spreads the rows of 8 consecutive threads over distinct bank quads).
constexpr int LROW = 52;

// Modes: see sph_build.cuh.
//
// STAGED (cap <= 48): a kept neighbour is one predicated shared-memory store
// into the thread's row -- no divergent branch around a global store in the
// candidate loop -- and the finished list leaves in 16-byte groups (a warp
// writes whole sectors); the rho/alpha pass reads the list back from shared
// memory.  Otherwise entries go straight to the global ELL list.
// With staging, shared memory limits an SM to 1024 / BS blocks (26.6 KB
// each at 128 threads); saying so lets the compiler use the registers that
// occupancy leaves (60 instead of 48 with spills: 529 -> 520 us at 1 M).
template <int MODE, int BS, bool STAGED>
__global__ void __launch_bounds__(BS, STAGED ? 1024 / BS : 1) k_build(DevScene s, GridGeom g, SolverConst c) {
    extern __shared__ int4 list_smem[];
    int* const row = reinterpret_cast<int*>(list_smem) + (STAGED ? threadIdx.x * LROW : 0);
    const int n = s.st->n_active;
    const int p = blockIdx.x * BS + threadIdx.x;
    int cnt = 0, over = 0;
    double ddiv = 0.0;  // MODE 4: this particle's Drho/Dt for the FP64 error
    const bool act = p < n;
    if (act) {
        const float4 pa = s.pos[p];
        const float4* __restrict__ P = s.pos;
        const float4* __restrict__ BP = s.bpos;
        const GridGeom G = s.nscenes > 1 ? s.b.geom[scene_of(pa)] : g;
        const int cx = cell_coord(pa.x, G.min[0], G.divisor);
        const int cy = cell_coord(pa.y, G.min[1], G.divisor);
        const int cz = cell_coord(pa.z, G.min[2], G.divisor);
        int* out = s.nbr;
        const size_t stride = (size_t)c.stride;
        const int cap = c.cap;
        // phase 1: candidate scan in the reference's order, append indices.
        // Every one of the 27 cells is scanned: skipping cells beyond the cut
        // per particle saves fewer tests than the per-cell test and the
        // divergence it causes among the lanes of one cell cost (measured).
        for (int dz = -1; dz <= 1; ++dz) {
            for (int dy = -1; dy <= 1; ++dy) {
                for (int dx = -1; dx <= 1; ++dx) {
                    const int x = cx + dx, y = cy + dy, z = cz + dz;
                    if (!cell_inside(G, x, y, z)) continue;
                    const int key = cell_key(G, x, y, z);
                    const int2 s0 = __ldg(s.cstart2 + key), s1 = __ldg(s.cstart2 + key + 1);
                    for (int q = s0.x; q < s1.x; ++q) {
                        const float4 pb = __ldg(P + q);
                        const float len2 = dis_square_rn(pa.x, pa.y, pa.z, pb.x, pb.y, pb.z);
                        const bool hit = len2 < c.h2cut && q != p;
                        if (STAGED) {
                            // cnt counts every hit; the first `cap` are kept
                            if (hit && cnt < cap) row[cnt] = q;
                            cnt += hit;
                        } else if (hit) {
                            if (cnt < cap) out[ell_index(stride, p, cnt++)] = q;
                            else ++over;
                        }
                    }
                    for (int q = s0.y; q < s1.y; ++q) {
                        const float4 pb = __ldg(BP + q);
                        const float len2 = dis_square_rn(pa.x, pa.y, pa.z, pb.x, pb.y, pb.z);
                        const bool hit = len2 < c.h2cut;
                        if (STAGED) {
                            if (hit && cnt < cap) row[cnt] = q | (int)BND_FLAG;
                            cnt += hit;
                        } else if (hit) {
                            if (cnt < cap) out[ell_index(stride, p, cnt++)] = q | (int)BND_FLAG;
                            else ++over;
                        }
                    }
                }
            }
        }
        if (STAGED) {
            over = cnt > cap ? cnt - cap : 0;
            cnt -= over;
            // the list in 16-byte groups (entries past the count are never
            // read: every sweep masks them)
            const int4* r4 = reinterpret_cast<const int4*>(row);
            int4* o4 = reinterpret_cast<int4*>(out);
            for (int gi = 0; gi < ((cnt + 3) >> 2); ++gi) o4[(size_t)gi * stride + p] = r4[gi];
        }
        s.ncount[p] = cnt;
        list_terms<MODE>(s, c, p, pa, cnt, ddiv, [&](int k, bool& bnd, float4& pb, float4& vb) {
            const unsigned e = STAGED ? (unsigned)row[k] : (unsigned)out[ell_index(stride, p, k)];
            bnd = (e & BND_FLAG) != 0u;
            // pv / bpv hold {the position (boundary: with its volume) of
            // pos / bpos, the velocity}
            if (build_has_div(MODE)) ld_record32((bnd ? s.bpv : s.pv) + 2 * (size_t)(e & BND_MASK), pb, vb);
            else pb = __ldg((bnd ? BP : P) + (e & BND_MASK));
        });
    }
    __shared__ int sh[BS / 32];
    int tot = block_sum_int<BS>(act ? cnt : 0, sh);
    int ov = block_sum_int<BS>(over, sh);
    int mx = block_max_int<BS>(act ? cnt : 0, sh);
    if (threadIdx.x == 0) {
        if (tot) atomicAdd(&s.st->nbr_total, (unsigned long long)tot);
        if (ov) { atomicAdd(&s.st->overflow, ov); atomicOr(&s.st->status, 8u); }
        if (mx) atomicMax(&s.st->max_nbrs, mx);
    }
    if (MODE == 4) {
        // the block's part of the iteration's FP64 sum of Drho/Dt (as
        // k_df_div_a; a batch, mode 5, reduces per scene in batch_decide)
        __shared__ double shd[BS / 32];
        const double bsum = block_sum_double<BS>(ddiv, shd);
        if (threadIdx.x == 0) s.partial[blockIdx.x] = bsum;
    }
}

__global__ void k_boundary_keys(const float4* bpos, int nb, GridGeom g, int* keys) {
    int i = blockIdx.x * NT + threadIdx.x;
    if (i >= nb) return;
    float4 p = bpos[i];
    int cx = cell_coord(p.x, g.min[0], g.divisor);
    int cy = cell_coord(p.y, g.min[1], g.divisor);
    int cz = cell_coord(p.z, g.min[2], g.divisor);
    keys[i] = cell_inside(g, cx, cy, cz) ? cell_key(g, cx, cy, cz) : -1;
}

// Boundary volume of a static rigid wall, SphBase::prepareSolidPartWeight
// (SphBase.cpp:766-813) with only boundary particles in the grid:
// V_b = 1 / (W(0, d) + sum over the (capped) boundary neighbour list of
// W(dis, (d_a + d_b)/2)).
__global__ void __launch_bounds__(128) k_boundary_volume(DevScene s, GridGeom g, float dpart, float h2cut, int cap,
                                                         int b0, int b1) {
    int p = b0 + blockIdx.x * 128 + threadIdx.x;
    if (p >= b1) return;
    float4 pa = s.bpos[p];
    int cx = cell_coord(pa.x, g.min[0], g.divisor);
    int cy = cell_coord(pa.y, g.min[1], g.divisor);
    int cz = cell_coord(pa.z, g.min[2], g.divisor);
    float h = dpart;
    float sum = ker_W_h(0.f, h);
    int cnt = 0;
    float hp = (dpart + dpart) / 2;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                int x = cx + dx, y = cy + dy, z = cz + dz;
                if (!cell_inside(g, x, y, z)) continue;
                int key = cell_key(g, x, y, z);
                int a = s.bcell_start[key], b = s.bcell_start[key + 1];
                for (int q = a; q < b; ++q) {
                    if (q == p) continue;
                    float4 pb = s.bpos[q];
                    float len2 = dis_square_rn(pa.x, pa.y, pa.z, pb.x, pb.y, pb.z);
                    if (len2 < h2cut && cnt < cap) {
                        ++cnt;
                        sum += ker_W_h(sqrtf(len2), hp);
                    }
                }
            }
    s.bpos[p].w = 1.f / sum;
}

// Reference-order transfers: gid is a permutation of [0, n) while no
// particle has been removed.
__global__ void k_to_ref_order(const float4* src, const int* gid, int n, float* dst3) {
    int p = blockIdx.x * NT + threadIdx.x;
    if (p >= n) return;
    float4 v = src[p];
    size_t g = (size_t)gid[p] * 3;
    dst3[g] = v.x;
    dst3[g + 1] = v.y;
    dst3[g + 2] = v.z;
}
// A host step's incoming state (reference order) against the sorted state
// whose lists are still valid: velocities go straight into the sorted
// arrays (vel and the velocity half of the force kernel's record); a
// position that differs from the device's sets *changed, and the caller
// then stages the positions and searches again.
__global__ void k_state_in(const float* xyz3, const float* vel3, const int* gid, int n, const float4* pos,
                           float4* vel, float4* prv, int* changed) {
    const int p = blockIdx.x * NT + threadIdx.x;
    int diff = 0;
    if (p < n) {
        const size_t g = (size_t)gid[p] * 3;
        const float4 x = pos[p];
        diff = x.x != xyz3[g] || x.y != xyz3[g + 1] || x.z != xyz3[g + 2];
        const float4 v = make_float4(vel3[g], vel3[g + 1], vel3[g + 2], 0.f);
        vel[p] = v;
        prv[2 * p + 1] = v;
    }
    if (__syncthreads_or(diff) && threadIdx.x == 0) atomicOr(changed, 1);
}

// Host state (reference order) against the sorted device state, bit for bit
// (positions and velocities): *differs set if any particle differs.  Reads
// only, so it can run while a step that has not yet re-sorted reads the same
// arrays.
__global__ void k_state_check(const float* xyz3, const float* vel3, const int* gid, int n, const float4* pos,
                              const float4* vel, int* differs) {
    const int p = blockIdx.x * NT + threadIdx.x;
    int diff = 0;
    if (p < n) {
        const size_t g = (size_t)gid[p] * 3;
        const float4 x = pos[p], v = vel[p];
        diff = (__float_as_int(x.x) != __float_as_int(xyz3[g])) | (__float_as_int(x.y) != __float_as_int(xyz3[g + 1])) |
               (__float_as_int(x.z) != __float_as_int(xyz3[g + 2])) | (__float_as_int(v.x) != __float_as_int(vel3[g])) |
               (__float_as_int(v.y) != __float_as_int(vel3[g + 1])) | (__float_as_int(v.z) != __float_as_int(vel3[g + 2]));
    }
    if (__syncthreads_or(diff) && threadIdx.x == 0) atomicOr(differs, 1);
}

// The positions the integration (k_hash, integrate mode) will write, in
// the same round-to-nearest operations, scattered into reference order:
// a host-buffer step copies them out while the rest of the step runs (the
// divergence loop changes velocities only).
__global__ void k_integrated_to_ref(DevScene s, float* out3) {
    const int n = s.st->n_active;
    const int i = blockIdx.x * NT + threadIdx.x;
    if (i >= n) return;
    float4 p = s.pos[i];
    const float dt = dt_of(s, p);
    const float4 v = s.pv[2 * i + 1];
    const size_t g = (size_t)s.gid[i] * 3;
    out3[g] = __fadd_rn(p.x, __fmul_rn(v.x, dt));
    out3[g + 1] = __fadd_rn(p.y, __fmul_rn(v.y, dt));
    out3[g + 2] = __fadd_rn(p.z, __fmul_rn(v.z, dt));
}

__global__ void k_from_ref_order(const float* src3, const int* gid, int n, float4* dst) {
    int p = blockIdx.x * NT + threadIdx.x;
    if (p >= n) return;
    size_t g = (size_t)gid[p] * 3;
    float4 v = dst[p];
    v.x = src3[g];
    v.y = src3[g + 1];
    v.z = src3[g + 2];
    dst[p] = v;
}
}  // namespace

static inline int nblk(int n, int nt) { return (n + nt - 1) / nt; }

void launch_to_ref_order(const float4* src, const int* gid, int n, float* dst3, cudaStream_t st) {
    if (n > 0) k_to_ref_order<<<nblk(n, NT), NT, 0, st>>>(src, gid, n, dst3);
}
void launch_state_in(const float* xyz3, const float* vel3, const int* gid, int n, const float4* pos, float4* vel,
                     float4* prv, int* changed, cudaStream_t st) {
    if (n > 0) k_state_in<<<nblk(n, NT), NT, 0, st>>>(xyz3, vel3, gid, n, pos, vel, prv, changed);
}
void launch_state_check(const float* xyz3, const float* vel3, const int* gid, int n, const float4* pos,
                        const float4* vel, int* differs, cudaStream_t st) {
    if (n > 0) k_state_check<<<nblk(n, NT), NT, 0, st>>>(xyz3, vel3, gid, n, pos, vel, differs);
}
void launch_integrated_to_ref(const DevScene& s, int n_max, float* out3, cudaStream_t st) {
    if (n_max > 0) k_integrated_to_ref<<<nblk(n_max, NT), NT, 0, st>>>(s, out3);
}
void launch_from_ref_order(const float* src3, const int* gid, int n, float4* dst, cudaStream_t st) {
    if (n > 0) k_from_ref_order<<<nblk(n, NT), NT, 0, st>>>(src3, gid, n, dst);
}


void launch_step_begin(const DevScene& s, cudaStream_t st) { k_step_begin<<<1, 1, 0, st>>>(s); }
void launch_call_begin(const DevScene& s, cudaStream_t st) { k_call_begin<<<1, 1, 0, st>>>(s); }
void launch_hash(const DevScene& s, const GridGeom& g, int integrate, int n_old, cudaStream_t st) {
    k_hash<<<nblk(n_old > 0 ? n_old : 1, NT), NT, 0, st>>>(s, g, integrate);
}

void launch_scan(const DevScene& s, const GridGeom& g, cudaStream_t st) {
    k_scan<<<1, SCAN_NT, 0, st>>>(s.cell_count, s.cell_start, g.nkeys + 1);
}

void launch_scatter_reorder(const DevScene& s, const GridGeom& g, int n_old, int carry, cudaStream_t st) {
    const int n = n_old > 0 ? n_old : 1;
    k_scatter<<<nblk(n > g.nkeys + 1 ? n : g.nkeys + 1, NT), NT, 0, st>>>(s, g.nkeys);
    k_rank_reorder<<<nblk(n, NT), NT, 0, st>>>(s, g.nkeys - 1, carry);
}

void launch_merge_starts(const DevScene& s, const GridGeom& g, cudaStream_t st) {
    k_merge_starts<<<nblk(g.nkeys + 1, NT), NT, 0, st>>>(s, g.nkeys);
}

template <int BS, bool STAGED>
static void launch_build_st(const DevScene& s, const GridGeom& g, const SolverConst& c, int mode, int nb,
                            cudaStream_t st) {
    const size_t sm = STAGED ? sizeof(int) * LROW * BS : 0;
    if (mode == 0) k_build<0, BS, STAGED><<<nb, BS, sm, st>>>(s, g, c);
    else if (mode == 1) k_build<1, BS, STAGED><<<nb, BS, sm, st>>>(s, g, c);
    else if (mode == 2) k_build<2, BS, STAGED><<<nb, BS, sm, st>>>(s, g, c);
    else if (mode == 4 && s.nscenes > 1) k_build<5, BS, STAGED><<<nb, BS, sm, st>>>(s, g, c);
    else if (mode == 4) k_build<4, BS, STAGED><<<nb, BS, sm, st>>>(s, g, c);
    else k_build<3, BS, STAGED><<<nb, BS, sm, st>>>(s, g, c);
}

template <int BS>
static void launch_build_bs(const DevScene& s, const GridGeom& g, const SolverConst& c, int mode, int n_max,
                            cudaStream_t st) {
    const int nb = nblk(n_max > 0 ? n_max : 1, BS);
    // staging needs the cap to fit a row and the rows to fit the default
    // 48 KB of dynamic shared memory (64 and 128 threads per block)
    if (c.cap <= LROW - 4 && BS * LROW * sizeof(int) <= 48 * 1024) launch_build_st<BS, true>(s, g, c, mode, nb, st);
    else launch_build_st<BS, false>(s, g, c, mode, nb, st);
}

// every block-size instantiation of the DFSPH list build (modes 1 and 4)
template <int BS, class F>
static void each_build_kernel_bs(F f) {
    f((const void*)k_build<1, BS, true>);
    f((const void*)k_build<1, BS, false>);
    f((const void*)k_build<4, BS, true>);
    f((const void*)k_build<4, BS, false>);
    f((const void*)k_build<5, BS, true>);
    f((const void*)k_build<5, BS, false>);
}
template <class F>
static void each_build_kernel(F f) {
    each_build_kernel_bs<64>(f);
    each_build_kernel_bs<128>(f);
    each_build_kernel_bs<256>(f);
}
// preferred shared-memory carveout of the DFSPH list build (percent; -1 =
// the driver's choice): the staged rows take shared memory from the L1 that
// caches the candidates' records
void set_build_carveout(int pct) {
    each_build_kernel([&](const void* k) { cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, pct); });
}
// loads every instantiation now (see preload_sweep_kernels)
void preload_build_kernels() {
    each_build_kernel([](const void* k) {
        cudaFuncAttributes a;
        cudaFuncGetAttributes(&a, k);
    });
}

void launch_build(const DevScene& s, const GridGeom& g, const SolverConst& c, int mode, int n_max, cudaStream_t st,
                  int bs) {
    if (c.build == 1 || (c.build == 2 && mode == 0)) {
        launch_warp_build(s, g, c, mode, n_max, st);
        return;
    }
    if (bs == 64) launch_build_bs<64>(s, g, c, mode, n_max, st);
    else if (bs == 256) launch_build_bs<256>(s, g, c, mode, n_max, st);
    else launch_build_bs<128>(s, g, c, mode, n_max, st);
}

int build_blocks(const SolverConst& c, int n_max, int bs) {
    if (c.build == 1) return warp_build_blocks(n_max);
    return nblk(n_max > 0 ? n_max : 1, bs == 64 || bs == 256 ? bs : 128);
}

void launch_boundary_keys(const float4* bpos, int nb, const GridGeom& g, int* keys, cudaStream_t st) {
    if (nb > 0) k_boundary_keys<<<nblk(nb, NT), NT, 0, st>>>(bpos, nb, g, keys);
}

void launch_boundary_volume(const DevScene& s, const GridGeom& g, float dpart, float h2cut, int cap, int b0, int b1,
                            cudaStream_t st) {
    if (b1 > b0) k_boundary_volume<<<nblk(b1 - b0, 128), 128, 0, st>>>(s, g, dpart, h2cut, cap, b0, b1);
}
