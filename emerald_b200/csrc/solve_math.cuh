// Per-particle sums of the five solvers, shared by the launch-per-phase
// kernels (solve_kernels.cu) and the resident solve kernel
// (resident_solve.cuh): both run these functions, so their results are the
// same operations in the same order, bit for bit.
//
// A function takes the particle's own values, and views of what it folds over:
// the fluid list (where entry k is read from: the arena, or a copy in shared
// memory), the boundary list, and the source of the neighbours' values. The
// views change where a value is read, not the value or its place in the sum.
#pragma once

#include "engine_types.cuh"
#include "kernels.cuh"
#include "sph_math.cuh"

namespace emerald {

// Block-level setup shared by the per-particle kernels. A tile belongs to
// one scene, so the scene checks are uniform across the block.
struct Ctx {
    int32_t s;
    uint32_t i;
    bool live;
};

__device__ __forceinline__ int iteration_cap(SceneParams const& P, int kind) {
    return kind == 0 ? P.iisph_max_iter : (kind == 3 ? 6 : P.dfsph_max_iter);
}

// The exit test of one solver iteration of a scene (kind 0: IISPH family,
// iisph.cpp:119-128; 1: DFSPH density, dfsph_p.cpp:113-133; 2: DFSPH
// divergence, :187-211; 3: PCISPH, pcisph.cpp:144-148), from the iteration's
// error sums; `iter` iterations ran before it. Returns whether the loop ends.
__device__ __forceinline__ bool loop_ends(SceneParams const& P, int kind, int iter,
                                          unsigned long long err_sum, uint32_t err_max) {
    float const mx = __uint_as_float(err_max);
    bool conv;
    if (kind == 0) {
        conv = iter > 1 && err_sum < P.sum_limit[0] && mx <= P.iisph_err_max;
    } else if (kind == 1) {
        conv = iter > 1 && err_sum < P.sum_limit[1] && mx <= P.dfsph_dens_max;
    } else if (kind == 2) {
        conv = iter > 0 && err_sum < P.sum_limit[2] && mx <= P.dfsph_div_max;
    } else {
        conv = iter > 1 && (mx / P.rho0) <= 0.01f;
    }
    return conv || iter + 1 >= iteration_cap(P, kind);
}

// The statistics of iteration `iter`, as the reference reports them; `ends`:
// it was the loop's last.
__device__ __forceinline__ void report_loop(SceneParams const& P, SceneState& S, int kind,
                                            int iter, unsigned long long err_sum,
                                            uint32_t err_max, bool ends) {
    double const n = static_cast<double>(1000ull * P.fluid_count);
    float const avg = P.fluid_count ? static_cast<float>(static_cast<double>(err_sum) / n) : 0.0f;
    float const mx = __uint_as_float(err_max);
    if (kind == 0) {
        S.stat_avg = avg;
        S.stat_max = mx;
    } else if (kind == 1 && iter > 1) {
        S.stat_avg = avg;
        S.stat_max = mx;
    } else if (kind == 2 && iter > 0) {
        S.stat_div_avg = avg;
        S.stat_div_max = mx;
    } else if (kind == 3 && iter > 1) {
        S.stat_max = mx / P.rho0;
    }
    if (ends) {
        if (kind == 2) {
            S.stat_div_iters = iter + 1;
        } else {
            S.stat_iters = iter + 1;
        }
    }
}

// The mean of the errors of iteration `iter`, reported beside the reference's
// metric (which drops each particle's error below 0.1%).
__device__ __forceinline__ void report_exact_mean(SceneParams const& P, SceneState& S, int kind,
                                                  int iter, double err_sum) {
    double const mean = P.fluid_count ? err_sum / static_cast<double>(P.fluid_count) : 0.0;
    if (kind == 1 && iter > 1) S.stat_avg_exact = mean;
    if (kind == 2 && iter > 0) S.stat_div_avg_exact = mean;
}

// --------------------------------------------------------- shared SPH sums

// Visits particle i's fluid list in list order, CH entries at a time: a
// chunk first loads its indices and kernel gradients, then every gathered
// neighbour value, then folds them into the sum in order. The loads of a
// chunk are independent, so they are in flight together; the sum is the
// same sequence of operations as a plain loop. The chunk of each kernel is
// a launch-time choice among 1, 4 and 8 (Tuning, set by the autotuner).
// These two are the chunks of callers that pass none (the IISPH final
// velocity update); the engine's DFSPH launches pass their Tuning's.
constexpr int kDivergenceChunk = 8;
constexpr int kPressureChunk = 4;

// Neighbours' values by arena slot (at) or by a list view's own code (local).
template <class T>
struct ArenaSource {
    T const* p;
    __device__ __forceinline__ T at(uint32_t j) const { return p[j]; }
};

// The fluid list of particle i in the arena: entry k at [k * stride + i].
struct ArenaList {
    static constexpr int kUnroll = 4;
    Arena const& a;
    uint32_t i;
    __device__ __forceinline__ uint32_t index(int k) const {
        return a.nf_idx[static_cast<size_t>(k) * a.stride + i];
    }
    __device__ __forceinline__ float2 gradient(int k) const {
        return a.nf_gw[static_cast<size_t>(k) * a.stride + i];
    }
    // f(neighbour's value, gradient, on) for entries [0, c), CH at a time; a
    // view may also call it past the list's end with on = false
    template <int CH, class Source, class Fold>
    __device__ __forceinline__ void fold(int c, Source const& src, Fold f) const {
        fold_range<CH>(0, c, src, f);
    }
    template <int CH, class Source, class Fold>
    __device__ __forceinline__ void fold_range(int k0, int c, Source const& src, Fold f) const {
        using T = decltype(src.at(0u));
        for (; k0 < c; k0 += CH) {
            uint32_t jj[CH];
            float2 gw[CH];
            T val[CH];
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                if (k0 + u < c) {
                    jj[u] = index(k0 + u);
                    gw[u] = gradient(k0 + u);
                }
            }
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                if (k0 + u < c) val[u] = src.at(jj[u]);
            }
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                if (k0 + u < c) f(val[u], gw[u], true);
            }
        }
    }
    // the neighbours' values alone (PCISPH recomputes its kernels)
    template <int CH, class Source, class Fold>
    __device__ __forceinline__ void fold_values(int c, Source const& src, Fold f) const {
        fold_values_range<CH>(0, c, src, f);
    }
    template <int CH, class Source, class Fold>
    __device__ __forceinline__ void fold_values_range(int k0, int c, Source const& src,
                                                      Fold f) const {
        using T = decltype(src.at(0u));
        for (; k0 < c; k0 += CH) {
            uint32_t jj[CH];
            T val[CH];
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                if (k0 + u < c) jj[u] = index(k0 + u);
            }
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                if (k0 + u < c) val[u] = src.at(jj[u]);
            }
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                if (k0 + u < c) f(val[u], true);
            }
        }
    }
};

// The boundary list of particle i in the arena: the mass rho0 V of entry k's
// boundary particle, its velocity, and the kernel gradient.
struct ArenaBoundary {
    static constexpr int kUnroll = 4;
    Arena const& a;
    uint32_t i;
    float rho0;
    __device__ __forceinline__ size_t entry(int k) const {
        return static_cast<size_t>(k) * a.stride + i;
    }
    __device__ __forceinline__ float mass(int k) const {
        return rho0 * a.vols[a.ns_idx[entry(k)]];
    }
    __device__ __forceinline__ float2 velocity(int k) const { return a.vs[a.ns_idx[entry(k)]]; }
    __device__ __forceinline__ float2 gradient(int k) const { return a.ns_gw[entry(k)]; }
};

// compute_densities (emerald/sph_common/density.cpp:10-73); with K each
// sum is Kahan-compensated.
template <bool K = false>
__device__ __forceinline__ float density_of(Arena const& a, SceneParams const& P, uint32_t i) {
    size_t const stride = a.stride;
    float const rho0 = P.rho0;
    float const fmass = rho0 * P.fluid_volume;
    SumF<K> d(P.fluid_volume * rho0 * P.w0);
    int const c = a.nf_cnt[i];
    #pragma unroll 4

    for (int k = 0; k < c; ++k) d.add(a.nf_w[k * stride + i] * fmass);
    float out = d.get();
    int const cs = a.ns_cnt[i];
    if (cs) {
        SumF<K> db;
        #pragma unroll 4

        for (int k = 0; k < cs; ++k) {
            size_t const e = k * stride + i;
            db.add(a.ns_w[e] * (rho0 * a.vols[a.ns_idx[e]]));
        }
        out += db.get();
    }
    return out;
}

// compute_divergences (emerald/sph_common/divergence.cpp:5-74).
// With K, the fluid and boundary terms go into one Kahan-compensated sum.
template <bool K = false, int CH = kDivergenceChunk, class List, class Boundary, class Source>
__device__ __forceinline__ float divergence_of(SceneParams const& P, int c, int cs, float2 vi,
                                               Source const& vels, List const& list,
                                               Boundary const& bnd) {
    float const fmass = P.rho0 * P.fluid_volume;
    SumF<K> sum;
    list.template fold<CH>(c, vels, [&](float2 vj, float2 g, bool on) {
        float2 const t = mul2p(sub2p(vi, vj), g);
        sum.add(fmass * (t.x + t.y), on);
    });
    if (K) {
        for (int k = 0; k < cs; ++k) {
            sum.add(bnd.mass(k) * dot2(sub2(vi, bnd.velocity(k)), bnd.gradient(k)));
        }
        return sum.get();
    }
    float d = sum.get();
    if (cs) {
        float db = 0.0f;
        #pragma unroll Boundary::kUnroll

        for (int k = 0; k < cs; ++k) {
            db += bnd.mass(k) * dot2(sub2(vi, bnd.velocity(k)), bnd.gradient(k));
        }
        d += db;
    }
    return d;
}

// apply_pressures_in_place (emerald/sph_common/pressure.cpp:9-80) for one
// particle, with q = safe_divide(p, rho^2) precomputed per particle. With K,
// each sum is Kahan-compensated.
template <bool K = false, int CH = kPressureChunk, class List, class Boundary, class Source>
__device__ __forceinline__ float2 apply_pressure_of(SceneParams const& P, int c, int cs, float2 v,
                                                    float qi, Source const& q, float dt,
                                                    List const& list, Boundary const& bnd) {
    float const neg_fmass = -(P.rho0 * P.fluid_volume);
    if (c) {
        SumF2<K> acc;
        list.template fold<CH>(c, q, [&](float qj, float2 g, bool on) {
            acc.add(scl2(neg_fmass * (qi + qj), g), on);
        });
        v = add2(v, scl2(dt, acc.get()));
    }
    if (cs) {
        SumF2<K> acc;
        #pragma unroll Boundary::kUnroll

        for (int k = 0; k < cs; ++k) acc.add(scl2(-bnd.mass(k) * qi, bnd.gradient(k)));
        v = add2(v, scl2(dt, acc.get()));
    }
    return v;
}

// compute_pressure_accelerations (emerald/sph_common/pressure.cpp:83-178);
// with K each sum is Kahan-compensated.
template <bool K = false, int CH = kPressureChunk, class List, class Boundary, class Source>
__device__ __forceinline__ float2 pressure_accel_of(SceneParams const& P, int c, int cs, float qi,
                                                    Source const& q, List const& list,
                                                    Boundary const& bnd) {
    float const neg_fmass = -(P.rho0 * P.fluid_volume);
    float2 out = mk2(0.0f, 0.0f);
    if (c) {
        SumF2<K> acc;
        list.template fold<CH>(c, q, [&](float qj, float2 g, bool on) {
            acc.add(scl2(neg_fmass * (qi + qj), g), on);
        });
        out = acc.get();
    }
    if (cs) {
        SumF2<K> acc;
        #pragma unroll Boundary::kUnroll

        for (int k = 0; k < cs; ++k) acc.add(scl2(-bnd.mass(k) * qi, bnd.gradient(k)));
        out = add2(out, acc.get());
    }
    return out;
}

// compute_all_external_forces (emerald/sph2d_box/forces.cpp:11-33) for one
// particle: the force starts at zero and takes the scene's terms in order,
// each with the reference function's own arithmetic; a scene driven by a
// host callback reads the callback's forces instead. v is the velocity at
// the point of the sub-step where the solver computes the forces.
__device__ __forceinline__ float2 external_force(Arena const& a, SceneParams const& P,
                                                 uint32_t i, float2 v) {
    if (P.force_array) return a.ext_f[i];
    float2 f = mk2(0.0f, 0.0f);
    for (int k = 0; k < P.force_count; ++k) {
        ForceTerm const t = P.force_terms[k];
        if (t.kind == kForceGravity) {
            // accumulate_gravity_forces (forces.cpp:63-71)
            f.y -= P.mass * t.a;
        } else if (t.kind == kForcePole) {
            // accumulate_constant_pole_attraction_forces (forces.cpp:85-101):
            // pull along the unit vector to the pole (Imath normalized(),
            // zero at the pole), plus the swirl (0, 0, magnitude / 8) x
            // (rN, 0) written out component by component.
            float2 const r = sub2(a.x[i], mk2(t.b, t.c));
            float const l = length2f(r);
            float2 const rn = (l == 0.0f) ? mk2(0.0f, 0.0f) : mk2(r.x / l, r.y / l);
            f = sub2(f, mk2(t.a * rn.x, t.a * rn.y));
            float const tz = 0.125f * t.a;
            float const zero = 0.0f;
            f = add2(f, mk2(zero * zero - tz * rn.y, tz * rn.x - zero * zero));
        } else if (t.kind == kForceDrag) {
            // accumulate_simple_drag_forces (forces.cpp:104-111)
            float const m = -t.a * t.b;
            f = add2(f, mk2(m * v.x, m * v.y));
        }
    }
    return f;
}

// integrate_velocities_in_place (dynamics.cpp:24-37) with the scene's
// external forces.
__device__ __forceinline__ float2 integrate_external(Arena const& a, SceneParams const& P,
                                                     uint32_t i, float2 v, float dt) {
    float2 const f = external_force(a, P, i, v);
    float const denom = P.rho0 * P.fluid_volume;
    float2 const numer = scl2(dt, f);
    if (safe_v(numer, denom)) v = add2(v, div2(numer, denom));
    return v;
}

// ------------------------------------------------------------------- DFSPH

// compute_densities + dfsph_p_compute_shared_coeffs (dfsph_p_ops.cpp:19-72).
// With K, the density and the two alpha sums are Kahan-compensated.
template <bool K, class List>
__device__ __forceinline__ void dfsph_density_alpha(Arena const& a, SceneParams const& P,
                                                    uint32_t i, int cf, int cs, List const& list,
                                                    float& rho, float& alpha) {
    size_t const stride = a.stride;
    float const rho0 = P.rho0;
    float const fvol = P.fluid_volume;
    float d = fvol * rho0 * P.w0;
    float2 sum = mk2(0.0f, 0.0f);
    float sdot = 0.0f;
    KahanF kd{d, 0.0f}, ksdot{0.0f, 0.0f};
    KahanF2 ksum{{0.0f, 0.0f}, {0.0f, 0.0f}};
    float const fmass = rho0 * fvol;
    float const fmass_a = fvol * rho0;
    #pragma unroll List::kUnroll

    for (int k = 0; k < cf; ++k) {
        size_t const e = k * stride + i;
        float2 const m = scl2(fmass_a, list.gradient(k));
        if (K) {
            kahan_add(kd, a.nf_w[e] * fmass);
            kahan_add(ksum, m);
            kahan_add(ksdot, dot2(m, m));
        } else {
            d += a.nf_w[e] * fmass;
            sum = add2(sum, m);
            sdot += dot2(m, m);
        }
    }
    if (cs) {
        float db = 0.0f;
        #pragma unroll 4

        for (int k = 0; k < cs; ++k) {
            size_t const e = k * stride + i;
            float const vs = a.vols[a.ns_idx[e]];
            if (K) {
                kahan_add(kd, a.ns_w[e] * (rho0 * vs));
                kahan_add(ksum, scl2(vs * rho0, a.ns_gw[e]));
            } else {
                db += a.ns_w[e] * (rho0 * vs);
                sum = add2(sum, scl2(vs * rho0, a.ns_gw[e]));
            }
        }
        if (!K) d += db;
    }
    if (K) {
        d = kd.s;
        sum = mk2(ksum.x.s, ksum.y.s);
        sdot = ksdot.s;
    }
    rho = d;
    alpha = 0.0f;
    if (cf + cs) {
        float const numer = sqrf(d);
        float const denom = dot2(sum, sum) + sdot;
        alpha = safe_f(numer, denom) ? numer / denom : 0.0f;
    }
}

// integrate_positions_in_place (dynamics.cpp:46-51). Compensated mode
// accumulates the positions in double and stores their float rounding.
// x_i += dt * v (+ shift): the reference's FP32 update, or for a
// compensated scene the FP64 accumulator (the positions the neighbour search
// takes its vectors from) rounded once into x_i. Every method's position
// update goes through here, so a compensated scene's FP64 positions stay
// current whichever method advances it.
__device__ __forceinline__ void advance_position(Arena const& a, SceneParams const& P,
                                                 uint32_t i, float dt, float2 v,
                                                 float2 shift = {0.0f, 0.0f}, bool shifted = false) {
    if (P.precision) {
        double2 x = a.x64[i];
        x.x += static_cast<double>(dt) * static_cast<double>(v.x);
        x.y += static_cast<double>(dt) * static_cast<double>(v.y);
        if (shifted) {
            x.x += static_cast<double>(shift.x);
            x.y += static_cast<double>(shift.y);
        }
        a.x64[i] = x;
        a.x[i] = mk2(static_cast<float>(x.x), static_cast<float>(x.y));
        return;
    }
    float2 const x = add2(a.x[i], scl2(dt, v));
    a.x[i] = shifted ? add2(x, shift) : x;
}

// A DFSPH pressure step of one particle: the pseudo pressure kappa, its
// kappa / rho^2, and the particle's error; for the density solve also rho*.
struct DfsphStep {
    float kappa, q, err, star;
};

// The errors of a particle with divergence d (dfsph_p.cpp:187-200), and with
// predicted density star (:134-148).
__device__ __forceinline__ float dfsph_divergence_error(SceneParams const& P, float dt, float d) {
    return d <= 0.0f ? 0.0f : (dt * d / P.rho0);
}
__device__ __forceinline__ float dfsph_density_error(SceneParams const& P, float star) {
    float const delta = star - P.rho0;
    return delta <= 0.0f ? 0.0f : (delta / P.rho0);
}

// dfsph_p_compute_divergence_pseudo_pressures (dfsph_p_ops.cpp:100-126) of a
// particle with divergence d, and its error.
__device__ __forceinline__ DfsphStep dfsph_divergence_step(SceneParams const& P, float dt,
                                                           float rho, float alpha, float d) {
    float kappa = 0.0f;
    if (!(d <= 0.0f)) {
        float const numer = d * alpha;
        kappa = safe_f(numer, dt) ? numer / dt : 0.0f;
    }
    return DfsphStep{kappa, p_over_rho2(kappa, rho), dfsph_divergence_error(P, dt, d), d};
}

// predict_density_stars (density.cpp:75-109) and
// dfsph_p_compute_density_pseudo_pressures (dfsph_p_ops.cpp:74-98) of a
// particle with divergence div, and its error.
__device__ __forceinline__ DfsphStep dfsph_density_step(SceneParams const& P, float dt, float rho,
                                                        float alpha, float div) {
    float const star = max_0x(rho + (dt * div));
    float const delta = star - P.rho0;
    float kappa = 0.0f;
    if (!(delta <= 0.0f)) {
        float const numer = delta * alpha;
        float const dd = sqrf(dt);
        kappa = safe_f(numer, dd) ? numer / dd : 0.0f;
    }
    return DfsphStep{kappa, p_over_rho2(kappa, rho), dfsph_density_error(P, star), star};
}

// -------------------------------------------------------------------- IISPH

// iisph_compute_diis (iisph_ops.cpp:20-90) of a particle with density rho.
// With K (compensated scenes), here and below, the sums are Kahan-compensated.
template <bool K, class List, class Boundary>
__device__ __forceinline__ float2 iisph_dii(SceneParams const& P, float dt, float rho, int cf,
                                            int cs, List const& list, Boundary const& bnd) {
    float const neg_dt2 = -sqrf(dt);
    float const denom = sqrf(rho);
    float2 dii = mk2(0.0f, 0.0f);
    if (cf) {
        float const fmass = P.rho0 * P.fluid_volume;
        SumF2<K> g;
        #pragma unroll List::kUnroll

        for (int k = 0; k < cf; ++k) g.add(scl2(fmass, list.gradient(k)));
        float2 const numer = scl2(neg_dt2, g.get());
        dii = safe_v(numer, denom) ? div2(numer, denom) : mk2(0.0f, 0.0f);
    }
    if (cs) {
        SumF2<K> g;
        #pragma unroll Boundary::kUnroll

        for (int k = 0; k < cs; ++k) g.add(scl2(bnd.mass(k), bnd.gradient(k)));
        float2 const numer = scl2(neg_dt2, g.get());
        dii = add2(dii, safe_v(numer, denom) ? div2(numer, denom) : mk2(0.0f, 0.0f));
    }
    return dii;
}

// Neighbour values the IISPH sums gather.
struct RhoV {
    float rho;
    float2 v;
};
struct IisphNeighbor {
    float rho, p;
    float2 sdp, dii;
};

// iisph_compute_aiis_and_density_stars (iisph_ops.cpp:92-200).
template <bool K, int CH = 4, class List, class Boundary, class Source>
__device__ __forceinline__ void iisph_aii(SceneParams const& P, float dt, float rho, float2 vi,
                                          float2 dii, int cf, int cs, Source const& src,
                                          List const& list, Boundary const& bnd, float& aii,
                                          float& star) {
    float const neg_dt2 = -sqrf(dt);
    aii = 0.0f;
    star = rho;
    if (cf) {
        float const mass = P.fluid_volume * P.rho0;
        SumF<K> af, dd;
        list.template fold<CH>(cf, src, [&](RhoV const& nb, float2 gw, bool on) {
            float2 const numer = scl2(neg_dt2 * mass, gw);
            float const denom = sqrf(nb.rho);
            if (on && safe_v(numer, denom)) {
                float2 const dji = neg2(div2(numer, denom));
                af.add(mass * dot2(sub2(dii, dji), gw));
            }
            dd.add(dt * mass * dot2(sub2(vi, nb.v), gw), on);
        });
        aii = af.get();
        star = rho + dd.get();
    }
    if (cs) {
        SumF<K> ab, dd;
        #pragma unroll Boundary::kUnroll

        for (int k = 0; k < cs; ++k) {
            float2 const gw = bnd.gradient(k);
            float const mass = bnd.mass(k);
            ab.add(mass * dot2(dii, gw));
            dd.add(dt * mass * dot2(sub2(vi, bnd.velocity(k)), gw));
        }
        aii += ab.get();
        star += dd.get();
    }
}

// iisph_compute_sum_dij_pjs (iisph_ops.cpp:202-235); the source gives
// (p_j, rho_j).
template <bool K, int CH, class List, class Source>
__device__ __forceinline__ float2 iisph_sum_dij(SceneParams const& P, float dt, int cf,
                                                Source const& p_rho, List const& list) {
    float const mass = P.fluid_volume * P.rho0;
    float const neg_dt2 = -sqrf(dt);
    SumF2<K> sum;
    list.template fold<CH>(cf, p_rho, [&](float2 prho, float2 g, bool on) {
        float2 const numer = scl2(neg_dt2 * mass * prho.x, g);
        float const denom = sqrf(prho.y);
        if (on && safe_v(numer, denom)) sum.add(div2(numer, denom));
    });
    return sum.get();
}

// iisph_compute_betas (iisph_ops.cpp:237-330) of a particle with pressure pi
// and sum of d_ij p_j si.
template <bool K, int CH, class List, class Boundary, class Source>
__device__ __forceinline__ float iisph_beta(SceneParams const& P, float dt, float pi, float2 si,
                                            int cf, int cs, Source const& src, List const& list,
                                            Boundary const& bnd) {
    float const neg_dt2 = -sqrf(dt);
    float beta = 0.0f;
    if (cf) {
        float const mass = P.rho0 * P.fluid_volume;
        SumF<K> bf;
        list.template fold<CH>(cf, src, [&](IisphNeighbor const& nb, float2 gw, bool on) {
            float2 const numer = scl2(neg_dt2 * mass, gw);
            float const denom = sqrf(nb.rho);
            float2 const dij = safe_v(numer, denom) ? div2(numer, denom) : mk2(0.0f, 0.0f);
            float2 const dji = neg2(dij);
            float2 const skni = sub2(nb.sdp, scl2(pi, dji));
            float2 const t = sub2(sub2(si, scl2(nb.p, nb.dii)), skni);
            bf.add(mass * dot2(t, gw), on);
        });
        beta = bf.get();
    }
    if (cs) {
        SumF<K> bb;
        #pragma unroll Boundary::kUnroll

        for (int k = 0; k < cs; ++k) bb.add(bnd.mass(k) * dot2(si, bnd.gradient(k)));
        beta += bb.get();
    }
    return beta;
}

// iisph_compute_new_pressures (iisph_ops.cpp:332-425) of a particle; sets
// `counted` where its error counts (a_ii != 0), and the scene's flag for an
// unsafe divide.
__device__ __forceinline__ float iisph_new_pressure(SceneParams const& P, SceneState* S, float pi,
                                                    float aii, float star, float beta, float& err,
                                                    bool& counted) {
    float out = pi;
    counted = false;
    if (aii != 0.0f) {
        float const numer = P.rho0 - star - beta;
        if (safe_f(numer, aii)) {
            err = max_0x(-(numer - (aii * pi)) / P.rho0);
            counted = true;
            out = max_0x(mix1(pi, numer / aii, P.iisph_omega));
        } else {
            atomicOr(&S->error, kErrNonFinite);
        }
    }
    return out;
}

// ------------------------------------------------- IISPH_AP / PSEUDO_AP

// iisph_ap_density_stars_and_diagonals (iisph_ap_ops.cpp:19-103) and the
// pseudo variant (iisph_pseudo_ap_ops.cpp:19-117).
template <bool K, int CH = 4, class List, class Boundary, class Source>
__device__ __forceinline__ void ap_diag(SceneParams const& P, float dt, float rho, float2 vi,
                                        int cf, int cs, int pseudo, Source const& vels,
                                        List const& list, Boundary const& bnd, float& aii,
                                        float& star) {
    if (!(cf + cs)) {
        star = rho;
        aii = 0.0f;
        return;
    }
    float const self_mass = P.fluid_volume * P.rho0;
    SumF2<K> sum_acc;
    SumF<K> sdot_acc, div_acc;
    float const fmass = P.fluid_volume * P.rho0;
    list.template fold<CH>(cf, vels, [&](float2 vj, float2 gw, bool on) {
        sum_acc.add(scl2(fmass, gw), on);
        sdot_acc.add(fmass * dot2(gw, gw), on);
        div_acc.add(fmass * dot2(sub2(vi, vj), gw), on);
    });
    #pragma unroll Boundary::kUnroll

    for (int k = 0; k < cs; ++k) {
        float2 const gw = bnd.gradient(k);
        float const mass = bnd.mass(k);
        sum_acc.add(scl2(mass, gw));
        div_acc.add(mass * dot2(sub2(vi, bnd.velocity(k)), gw));
    }
    float2 const sum = sum_acc.get();
    float const sdot = sdot_acc.get();
    float const div = div_acc.get();
    float const denom = sqrf(rho);
    float const numer = pseudo ? -(dot2(sum, sum) + self_mass * sdot)
                               : -sqrf(dt) * (dot2(sum, sum) + self_mass * sdot);
    aii = safe_f(numer, denom) ? numer / denom : 0.0f;
    star = rho + dt * div;
}

// One particle's pressure update of a Jacobi iteration
// (iisph_ap_iterate_pressures_in_place, iisph_ap_ops.cpp:105-194, and the
// pseudo variant, iisph_pseudo_ap_ops.cpp:226-323) from its pressure
// acceleration ai and its neighbours'; sets `counted` where its error counts.
template <bool K, int CH = 4, class List, class Boundary, class Source>
__device__ __forceinline__ float ap_iterate(SceneParams const& P, float dt, int cf, int cs,
                                            int pseudo, float diag, float star, float old,
                                            float2 ai, Source const& accs, List const& list,
                                            Boundary const& bnd, float& err, bool& counted) {
    float const rho0 = P.rho0;
    counted = false;
    if ((!cf && !cs) || (pseudo && diag == 0.0f)) return 0.0f;
    SumF<K> sum;
    float const fmass = rho0 * P.fluid_volume;
    list.template fold<CH>(cf, accs, [&](float2 aj, float2 g, bool on) {
        float2 const t = mul2p(sub2p(ai, aj), g);
        sum.add(fmass * (t.x + t.y), on);
    });
    #pragma unroll Boundary::kUnroll

    for (int k = 0; k < cs; ++k) sum.add(bnd.mass(k) * dot2(ai, bnd.gradient(k)));
    float api = sum.get();
    if (!pseudo) api *= sqrf(dt);
    float const source = rho0 - star;
    float const r = api - source;
    err = max_0x(safe_f(r, rho0) ? r / rho0 : 0.0f);
    counted = true;
    float const numer = P.iisph_omega * (source - api);
    return max_0x(old + (safe_f(numer, diag) ? numer / diag : 0.0f));
}

// The integration after the final pressure accelerations: iisph_ap.cpp:138-153
// (integrate_velocities_and_positions_in_place, dynamics.cpp:53-63) or
// iisph_pseudo_ap_integrate_velocities_and_positions_in_place
// (iisph_pseudo_ap_ops.cpp:325-343).
__device__ __forceinline__ void ap_integrate(Arena const& a, SceneParams const& P, uint32_t i,
                                             float dt, float2 v, float2 acc, int pseudo) {
    if (!pseudo) {
        v = add2(v, scl2(dt, acc));
        a.v[i] = v;
        advance_position(a, P, i, dt, v);
    } else {
        advance_position(a, P, i, dt, v, acc, true);
        if (safe_v(v, dt)) a.v[i] = add2(v, div2(acc, dt));
    }
}

// ------------------------------------------------------------------- PCISPH

// Velocity from external forces only (pcisph.cpp:54-65).
__device__ __forceinline__ float2 pc_external_velocity(Arena const& a, SceneParams const& P,
                                                       uint32_t i, float dt, float2 v) {
    float const mult = dt / P.mass;
    return add2(v, scl2(mult, external_force(a, P, i, v)));
}

// Predicted velocity of predictor pass `iter` (pcisph.cpp:72-88).
__device__ __forceinline__ float2 pc_predicted_velocity(SceneParams const& P, float dt, int iter,
                                                        float2 vext, float2 force) {
    return iter > 0 ? add2(vext, scl2(dt / P.mass, force)) : vext;
}

// Densities at the predicted positions with the kernel values recomputed
// (compute_neighbor_distances_and_vectors_to + compute_neighbor_kernels,
// neighborhoods_from_state.cpp:103-128), pcisph_compute_densities and
// pcisph_accumulate_density_from_solids (pcisph_ops.cpp:18-60).
template <bool K, int CH = 4, class List, class Source>
__device__ __forceinline__ float pc_density_of(Arena const& a, SceneParams const& P, uint32_t i,
                                               float2 pos, int cf, int cs, Source const& xs,
                                               List const& list) {
    size_t const stride = a.stride;
    float const h = P.support;
    SumF<K> ws(P.w0);
    list.template fold_values<CH>(cf, xs, [&](float2 xj, bool on) {
        if (on) ws.add(kernel_w(length2f(sub2(xj, pos)), h));
    });
    float d = P.mass * ws.get();
    if (cs) {
        SumF<K> vf;
        #pragma unroll 4

        for (int k = 0; k < cs; ++k) {
            uint32_t const j = a.ns_idx[k * stride + i];
            vf.add(a.vols[j] * kernel_w(length2f(sub2(a.xs[j], pos)), h));
        }
        d += P.rho0 * vf.get();
    }
    return d;
}

// The pressure of a particle with predicted density d
// (pcisph_update_pressures, pcisph_ops.cpp:60-76), from its pressure so far.
__device__ __forceinline__ float pc_pressure(SceneParams const& P, float p, float d) {
    return p + max_x0(d - P.rho0) / P.pcisph_denom;
}

// Neighbour values the PCISPH forces gather.
struct PcNeighbor {
    float2 x, v;
    float rho, q;
};

// pcisph_accumulate_pressure_forces and ..._from_solids (pcisph_ops.cpp:78-178)
// on the fixed neighbour lists at the predicted positions. `p` is the
// particle's pressure, `self` its predicted state.
template <bool K, int CH = 2, class List, class Source>
__device__ __forceinline__ float2 pc_forces(Arena const& a, SceneParams const& P, uint32_t i,
                                            PcNeighbor const& self, float p, int cf, int cs,
                                            Source const& src, List const& list) {
    size_t const stride = a.stride;
    float const h = P.support;
    float const m = P.mass;
    float const N2 = 0.01f * h * h;
    float2 f = mk2(0.0f, 0.0f);
    if (cf) {
        SumF2<K> pf;
        list.template fold_values<CH>(cf, src, [&](PcNeighbor const& nb, bool on) {
            if (!on) return;
            float2 const vto = sub2(nb.x, self.x);
            float const dist = length2f(vto);
            float2 const gw = kernel_grad_w(neg2(vto), h);
            pf.add(scl2(self.q + nb.q, gw));
            float2 const dv = sub2(nb.v, self.v);
            float const dvr = dot2(vto, dv);
            if (dvr < 0.0f) {
                float const mu = h * dvr / (dist + N2);
                float const den = (self.rho + nb.rho) / 2.0f;
                pf.add(scl2(((-1.0f * P.viscosity * mu) + (2.0f * sqrf(mu))) / den, gw));
            }
        });
        f = add2(f, scl2(-(m * m), pf.get()));
    }
    if (cs) {
        float const pors = p / sqrf(self.rho);
        SumF2<K> vg;
        #pragma unroll 4

        for (int k = 0; k < cs; ++k) {
            uint32_t const j = a.ns_idx[k * stride + i];
            float2 const gw = kernel_grad_w(neg2(sub2(a.xs[j], self.x)), h);
            vg.add(scl2(a.vols[j], gw));
        }
        f = add2(f, scl2(-m * P.rho0 * pors, vg.get()));
    }
    return f;
}

}  // namespace emerald
