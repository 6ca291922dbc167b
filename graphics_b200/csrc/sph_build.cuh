// sph_build.cuh -- the terms the neighbour-list build computes over a list it
// has just written, shared by the build kernels (sph_grid.cu, sph_warp.cu).
#pragma once
#include "sph_kernels.cuh"

// mode 0: neighbour lists only; 1: + DFSPH rho and alpha
// (DF_constantDensitySolverFirst, DFSPH.cpp:84-193); 2: + WCSPH rho and Tait
// pressure (WcSph::wc_computePressure, WcSph.cpp:99-153); 3: + IISph
// sphDensity, gamma, sphVolume and alpha (IISph.cpp:100-402); 4: mode 1 and,
// over the same list in the same pass, the first sweep A of the divergence
// loop that follows the neighbour search (DFSPH.cpp:795-835: Drho/Dt, its
// clamp, kappa_v, the FP64 error sum) -- the loop then starts with its
// velocity update (the per-pair term is div_term, the one the separate sweep
// uses, so the results are the same bit for bit); 5: mode 4 in a batch (each
// scene's own dt; the loop decisions reduce per scene).
constexpr bool build_has_div(int mode) { return mode == 4 || mode == 5; }

// The sums a mode takes over a list, in list order, each a chain of
// acc = fma(u, v, acc): 1: density, sum m gradW (3), sum |m gradW|^2 over
// fluid; 2: density, in blocks of DENS_BLOCK entries whose sums are added in
// turn, since the pressure is its seventh power (error against FP64, 30 blocks of
// 1 000 particles: density 1.12e-7 rms so, 1.30e-7 in one chain; the pressures'
// largest 4.3e-6 against 5.6e-6); 3: density, gamma, sphVolume, sum V gradW (3),
// sum V^2 |gradW|^2 / m over fluid; 4 and 5: mode 1's and the divergence sum.
constexpr int DENS_BLOCK = 8;
template <int MODE>
struct BuildSums {
    static constexpr int N = MODE == 2 ? 1 : MODE == 3 ? 7 : build_has_div(MODE) ? 6 : 5;
    float v[N];
};
template <int MODE>
__device__ __forceinline__ void sums_begin(const SolverConst& c, float4 pa, BuildSums<MODE>& a) {
    const int ph = phase_of(pa);
#pragma unroll
    for (int i = 0; i < BuildSums<MODE>::N; ++i) a.v[i] = 0.f;
    if (MODE == 3) {
        const float Va = c.iv_V, w0 = c.kd.theta;  // W(0, d)
        a.v[0] = w0 * c.iv_m[ph];
        a.v[1] = Va * w0;
        a.v[2] = (float)((double)w0 * (double)Va * (double)Va);
    } else {
        a.v[0] = ker_W(c.k, 0.f) * c.fm_ph[ph];
    }
}
// One entry's factors u, v of every sum: its kind, its position (w: a
// boundary particle's volume, a fluid particle's phase bits) and, where the
// mode has the divergence sweep, its velocity.
template <int MODE>
__device__ __forceinline__ void pair_terms(const SolverConst& c, float4 pa, float4 va, bool bnd, float4 pb, float4 vb,
                                           BuildSums<MODE>& u, BuildSums<MODE>& v) {
    const int ph = phase_of(pa);
    const float rho0 = c.rho0_ph[ph];
    const float xx = pa.x - pb.x, xy = pa.y - pb.y, xz = pa.z - pb.z;
    const float len2 = dis_square_rn(pa.x, pa.y, pa.z, pb.x, pb.y, pb.z);
    float w, f;
    if (MODE == 3) {
        // IISph: sphDensity (DF_prepareAttribute, IISph.cpp:127-170) and
        // VF_prepareAttribute (IISph.cpp:309-402) over the stored list,
        // per-pair h = (d_a + d_b)/2 = d (one diameter for all particles)
        kernel_pair_rn(c.kd, len2, w, f);
        const float Va = c.iv_V;
        const float Vb = bnd ? pb.w : Va;
        u.v[0] = bnd ? rho0 * Vb : c.iv_m[phase_of(pb)];
        u.v[1] = Vb;
        u.v[2] = Va * Vb;
        v.v[0] = v.v[1] = v.v[2] = w;
        const float fv = f * Vb;
        u.v[3] = xx;
        u.v[4] = xy;
        u.v[5] = xz;
        v.v[3] = v.v[4] = v.v[5] = fv;
        // V_b^2 |gradW|^2 / m_b: fluid neighbours only (boundary terms
        // belong to dynamic solids, IISph.cpp:386-393)
        u.v[6] = bnd ? 0.f : fv * fv;
        v.v[6] = bnd ? 0.f : len2 / c.iv_m[phase_of(pb)];
        return;
    }
    kernel_pair(c.k, len2, w, f);
    const float m = bnd ? rho0 * pb.w : c.fm_ph[ph];
    u.v[0] = m;
    v.v[0] = w;
    if (MODE == 1 || build_has_div(MODE)) {
        const float fm = f * m;
        u.v[1] = xx;
        u.v[2] = xy;
        u.v[3] = xz;
        v.v[1] = v.v[2] = v.v[3] = fm;
        const float t = bnd ? 0.f : fm * sqrtf(len2);  // |gradW| m, fluid only (DFSPH.cpp:161)
        u.v[4] = v.v[4] = t;
    }
    if (build_has_div(MODE)) div_pair(c, pa, va, pb, vb, bnd, u.v[5], v.v[5]);
}
// What the mode writes for particle p from its sums; the particle's Drho/Dt
// (modes 4 and 5).
template <int MODE>
__device__ __forceinline__ double sums_finish(const DevScene& s, const SolverConst& c, int p, float4 pa,
                                              const BuildSums<MODE>& a) {
    const int ph = phase_of(pa);
    const float rho0 = c.rho0_ph[ph];
    const float density = a.v[0];
    if (MODE == 3) {
        float al = ((a.v[3] * a.v[3] + a.v[4] * a.v[4] + a.v[5] * a.v[5]) / c.iv_m[ph] + a.v[6]) / a.v[1];
        if (al < 1.0e-10f) al = 1.0e-10f;
        s.ivs[p] = make_float4(a.v[1], a.v[2], 1.f / al, density);
        return 0.0;
    }
    s.rho[p] = density;
    if (MODE == 2) {
        // Tait, WcSph.cpp:142-146 (NEGLECT_NEGATIVE_PRESSURE)
        float pr = c.wc_B * (powf(density / rho0, c.wc_gamma) - 1.f);
        if (pr < 0.f) pr = 0.f;
        s.kr[p] = pr;
        wc_record(s, p, pa, s.vel[p], density, pr);
        return 0.0;
    }
    s.prv[2 * p] = make_float4(pa.x, pa.y, pa.z, density);
    float al = a.v[1] * a.v[1] + a.v[2] * a.v[2] + a.v[3] * a.v[3] + a.v[4];
    if (al < 1.0e-6f) al = 1.0e-6f;
    const float alpha = density / al;
    s.alpha[p] = alpha;
    if (!build_has_div(MODE)) return 0.0;
    // the divergence loop's first sweep A, as k_df_div_a
    const float dt = MODE == 5 ? s.b.dt[scene_of(pa)] : *s.dt;
    float dd = a.v[5];
    if (dd < 0.f || (density + dd * dt) < c.rho0) dd = 0.f;  // DFSPH.cpp:829-832
    const float kv = dd * alpha / dt;                         // DFSPH.cpp:835
    s.pk[p] = make_float4(pa.x, pa.y, pa.z, kv / density);
    s.kappav[p] = kv;
    s.aux1[p] = dd;
    return (double)dd;
}

// The mode's terms of particle p over its cnt list entries, by one thread.
// fetch(k, bnd, pb, vb): entry k as pair_terms takes it.  ddiv: the
// particle's Drho/Dt (modes 4 and 5).
template <int MODE, class Fetch>
__device__ __forceinline__ void list_terms(const DevScene& s, const SolverConst& c, int p, float4 pa, int cnt,
                                           double& ddiv, Fetch&& fetch) {
    if (MODE == 0) return;
    BuildSums<MODE> a;
    sums_begin<MODE>(c, pa, a);
    const float4 va = build_has_div(MODE) ? s.pv[2 * p + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
    auto entries = [&](int k, int end, BuildSums<MODE>& t) {
#pragma unroll 4
        for (; k < end; ++k) {
            bool bnd;
            float4 pb, vb;
            fetch(k, bnd, pb, vb);
            BuildSums<MODE> u, v;
            pair_terms<MODE>(c, pa, va, bnd, pb, vb, u, v);
#pragma unroll
            for (int i = 0; i < BuildSums<MODE>::N; ++i) t.v[i] = fmaf(u.v[i], v.v[i], t.v[i]);
        }
    };
    if (MODE == 2) {
        // (whole blocks first: of a known length, so that their loads go together)
        int k0 = 0;
        for (; k0 + DENS_BLOCK <= cnt; k0 += DENS_BLOCK) {
            BuildSums<MODE> t;
            t.v[0] = 0.f;
            entries(k0, k0 + DENS_BLOCK, t);
            a.v[0] += t.v[0];
        }
        BuildSums<MODE> t;
        t.v[0] = 0.f;
        entries(k0, cnt, t);
        a.v[0] += t.v[0];
    } else {
        entries(0, cnt, a);
    }
    ddiv = sums_finish<MODE>(s, c, p, pa, a);
}
