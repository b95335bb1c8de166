// The sm_103a kernels of the FP64 2D shallow-water split-form stage.
//
// This file is compiled twice (kernels_fast.cu, kernels_exact.cu) into two
// namespaces: DGSWE_FAST = 1 lets the compiler contract multiply-adds into
// FMA (-fmad=true), evaluates the Manning rate without divisions, and does
// the wet elements' volume term, the wet faces' fluxes and every square root
// and quotient in 62-bit fixed point on the integer pipes (fixed64.hpp: an
// FP64 warp instruction holds its pipe for 64 cycles here, the time of some
// thirty integer multiply-adds); 0 keeps every multiply and add separately
// rounded FP64 (-fmad=false) and follows the reference's arithmetic, its cube
// root included. A wet element's sums have one last place for all its nodes in
// fixed point; where that is further from a node's result than FP64's rounding,
// FP64 takes the element or the node (fixed64.hpp), so that no node's error is
// above FP64's.
//
// Kernels of one stage (one RK stage of every element):
//  - face_kernel: the numerical flux F* of every interior edge node once,
//    from the edge's left side with that side's normal (the reference's
//    edge_fluxes, src/solver/rhs/swe_2d_split_form.rs:580-616), and of every
//    boundary face node (wall or characteristic open boundary), stored per
//    element face node as each side sees it;
//  - stage_kernel<N1>: per element, the split-form volume term (flux
//    differencing on wet elements, subcell finite volumes on elements with a
//    node shallower than the subcell depth), the face fluxes lifted by each
//    face node's sJ·LIFT (a multiply-add in the stage, not a multiply in
//    the face pass), 1/J,
//    Coriolis, the Shu–Osher combination, the point-implicit damping and the
//    wet/dry correction or the accumulation (the reference's fused
//    stage_where, src/physics/builder.rs:652-737), and the node velocities
//    the next stage reads;
//  - with DGSWE_FAST, general_kernel<N1>: the same for the elements that fixed
//    point leaves (subcells with water, nodes that FP64 is closer to), listed by
//    stage_kernel or, beside the face pass, by shallow_list_kernel.
// Per step: dt_min_kernel<N1> (the smallest element step; dt_kernel<N1> where
// every element's is asked for) and three one-thread kernels that run the
// step's clock on the device, so that a whole step is one CUDA graph. Once
// per handle, fixed_tables_kernel (the mesh's fixed-point tables) and
// sub_metric_kernel (the subcells' geometry).
//
// The volume and surface terms use the summation-by-parts identity of the
// GLL operators: at a line end the volume term's 2·D₀₀·F(q)·Ja and the
// surface term's LIFT·sJ·F(q)·n are equal and opposite (2D₀₀ = −1/w₀,
// LIFT = 1/w₀ on the face node, sJ·n = −Ja), so neither is evaluated: the
// interior diagonal of D is zero, and what remains is the pair fluxes and
// −LIFT·sJ·F*. The same holds for the subcells' end fluxes. The result
// differs from the reference's by rounding only.

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "device.hpp"
#include "fp64_bits.hpp"
#include "point.cuh"

namespace dgswe {
namespace DGSWE_NS {

enum StageMode { kRhsOnly = 0, kPost = 1, kAccumulate = 2 };

__device__ __forceinline__ Q load_q(const DevBuf& in, const DevTables& T, const Physics& P,
                                    int64_t g) {
    Q q;
    q.h = in.h[g];
    q.hu = in.hu[g];
    q.hv = in.hv[g];
    q.u = in.u[g];
    q.v = in.v[g];
    q.b = P.has_bed ? T.bed[g] : 0.0;
    return q;
}

__device__ __forceinline__ Sd load_side(const DevBuf& in, const DevTables& T, const Physics& P,
                                        int64_t g) {
    return {in.h[g], in.u[g], in.v[g], P.has_bed ? T.bed[g] : 0.0};
}

struct FacePair {
    F3 a, b;
};

// hydro_hll of a face node along its geometry. With DGSWE_FAST, where the
// interior faces mostly take fixed point, this is a call: the rest (exponents
// out of range, some films near the datum: fx::kNoScale) then runs the same
// instructions in every face kernel, the multiply-adds contracted alike, and its
// registers are not the kernels'.
#if DGSWE_FAST
__device__ __noinline__
#else
__device__ __forceinline__
#endif
    FacePair face_hll(Sd qa, Sd qb, const double* geo, double g, double sqrt_g, double half_g,
                      double h_min) {
    FacePair f;
    hydro_hll(qa, qb, geo[0], geo[1], geo[2], geo[3], geo[4], g, sqrt_g, half_g, h_min, f.a, f.b);
    return f;
}

#if DGSWE_FAST
__device__ __noinline__ FacePair face_dry(Sd qa, Sd qb, const double* geo, double g, double half_g,
                                          double h_min) {
    FacePair f;
    hydro_dry(qa, qb, geo[0], geo[1], geo[3], geo[4], g, half_g, h_min, f.a, f.b);
    return f;
}

// The flux of two sides along m = norm·(nx, ny): in fixed point, or the rest
__device__ __forceinline__ FacePair face_pair(const DevTables& T, const Sd& qa, const Sd& qb,
                                              const double* geo, double g, double sqrt_g,
                                              double half_g, double h_min) {
    fx::FaceFlux f;
    const fx::FaceCase got =
        T.fx_face.usable ? fx::face_flux(qa, qb, geo, T.fx_face, h_min, f) : fx::kNoScale;
    if (got == fx::kDone) return {{f.h, f.hu_a, f.hv_a}, {f.h, f.hu_b, f.hv_b}};
    if (got == fx::kBothDry) return face_dry(qa, qb, geo, g, half_g, h_min);
    return face_hll(qa, qb, geo, g, sqrt_g, half_g, h_min);
}
#endif

// An element's stage in a multirate pass (element_stage,
// src/time/multirate.rs:169-200), every operation rounded on its own as the
// reference's are (no contraction): its substep's start time and step, the
// Shu–Osher weights, and for the last stage the weight of its sum (the mean
// of the substep's 2^(rate − level) blocks, restarted where the substep
// starts). dt/2^level and 1/2^(rate − level) are exact.
__device__ __forceinline__ StageArgs lts_stage(const LtsPass& p, int64_t k) {
    const int l = p.level[k];
    const double inv_2l = __longlong_as_double((long long)(1023 - l) << 52);  // 2^-l
    const double dt_l = __dmul_rn(p.dt, inv_2l);
    const long long q = (long long)p.substep >> (p.finest - l);
    const double t_k = __dadd_rn(p.t, __dmul_rn((double)q, dt_l));
    StageArgs a;
    a.time = __dadd_rn(t_k, __dmul_rn(p.c, dt_l));
    a.a = p.start;
    a.b = p.input;
    a.c = __dmul_rn(p.beta, dt_l);
    a.w = 1.0;
    a.keep = 0.0;
    if (p.last) {
        const int blocks = p.rate[k] - l;
        a.w = __longlong_as_double((long long)(1023 - blocks) << 52);  // 1/2^(rate − level)
        a.keep = l >= p.depth ? 0.0 : 1.0;
    }
    return a;
}

// The interface flux of the other split forms (EntropyStable / EntropyConservative):
// F#·n (+ dissipation) with the bed interface term per side
// (src/solver/rhs/swe_2d_split_form.rs:639-650, src/flux/swe_2d_entropy.rs:166-205)
__device__ void entropy_surface(const Q& qa, const Q& qb, double nx, double ny, const Physics& P,
                                F3& fa, F3& fb) {
    const double g = P.g;
    F3 s = wflux(qa, qb, nx, ny, g);
    if (P.formulation == kEntropyStable) {
        const double sp_i = fabs(qa.u * nx + qa.v * ny) + sqrt(g * fmax(qa.h, 0.0));
        const double sp_e = fabs(qb.u * nx + qb.v * ny) + sqrt(g * fmax(qb.h, 0.0));
        const double scale = -0.5 * fmax(sp_i, sp_e);
        const double jump = (qb.h + qb.b) - (qa.h + qa.b);
        const double h_avg = 0.5 * (qa.h + qb.h), u_avg = 0.5 * (qa.u + qb.u),
                     v_avg = 0.5 * (qa.v + qb.v);
        s.h = s.h + scale * jump;
        s.hu = s.hu + scale * (u_avg * jump + h_avg * (qb.u - qa.u));
        s.hv = s.hv + scale * (v_avg * jump + h_avg * (qb.v - qa.v));
    }
    const double fa_b = 0.5 * g * qa.h * (qb.b - qa.b);
    const double fb_b = 0.5 * g * qb.h * (qa.b - qb.b);
    fa = {s.h + 0.0, s.hu + fa_b * nx, s.hv + fa_b * ny};
    fb = {-s.h + 0.0, -s.hu + fb_b * (-nx), -s.hv + fb_b * (-ny)};
}

// The nesting relaxation band's source at the stage's input, per band node
// (NestingRelaxation2D::add_element and relaxation_source,
// src/boundary/ocean_nesting.rs:955-1030), into T.rx_src at its element's
// stage time (in a multirate pass, the element's own)
template <bool LISTED>
__global__ void __launch_bounds__(256) relax_kernel(DevTables T, Physics P, DevBuf in,
                                                    const StepCtl* ctl, int slot, LtsPass lp) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= T.rx_n) return;
    const int64_t g = T.rx_node[b];
    const int64_t k = g / P.nn;
    const int32_t s = T.rx_slot[b];
    const int64_t nv = T.K * P.nn;
    double sh = 0.0, shu = 0.0, shv = 0.0;
    const double h = in.h[g], w = T.rx_weight[s];
    if (fp::gt0(w) && !fp::lt(h, T.rx_wet)) {
        const int member = T.elem_member ? T.elem_member[k] : 0;
        const double t = LISTED ? lts_stage(lp, k).time : ctl[member].stage[slot].time;
        const double bed = P.has_bed ? T.bed[g] : 0.0;
        double eta, u, v;
        bool has_uv;
        parent_state_at(T.rx_times, T.rx_n_times, T.rx_cubic, T.rx_values + (int64_t)s * T.rx_n_times * 3,
                        t, T.rx_ramp, T.rx_ref_level, T.rx_velocity, T.rx_max_ratio, T.rx_depth[s],
                        bed, eta, u, v, has_uv);
        const double hp = eta - bed;
        if (!fp::lt(hp, T.rx_wet)) {
            const double gamma = w * T.rx_rate;
            const double hu = in.hu[g], hv = in.hv[g];
            if (!has_uv) {
                u = hu / h;
                v = hv / h;
            }
            const double dh = T.rx_momentum_only ? 0.0 : hp - h;
            const double depth = T.rx_momentum_only ? h : hp;
            sh = gamma * dh;
            shu = gamma * (depth * u - hu);
            shv = gamma * (depth * v - hv);
        }
    }
    if (T.at_source) {  // added to the weather's source of this pass
        T.rx_src[g] += sh;
        T.rx_src[nv + g] += shu;
        T.rx_src[2 * nv + g] += shv;
    } else {
        T.rx_src[g] = sh;
        T.rx_src[nv + g] = shu;
        T.rx_src[2 * nv + g] = shv;
    }
}

// The weather's momentum source at the stage's input
// (GriddedAtmosphere2D::add_element, src/source/swe_2d/gridded_atmosphere.rs:698-729),
// per node of every element (LISTED: of the pass's elements) at its
// element's stage time, into T.rx_src; the relaxation band's kernel,
// launched after it, adds the band's
template <bool LISTED>
__global__ void __launch_bounds__(256) atmos_kernel(DevTables T, Physics P, DevBuf in,
                                                    const StepCtl* ctl, int slot, LtsPass lp) {
    // one stage time for every node of a global stage: its time weights and
    // ramp once per block, in shared memory
    __shared__ int s_idx[2], s_len;
    __shared__ double s_w[2], s_ramp;
    if (!LISTED) {
        if (threadIdx.x == 0) {
            const double t = ctl[0].stage[slot].time;
            int idx[2];
            double w[2];
            s_len = weather_weights(T.at_times, T.at_n_times, T.at_epoch + t, idx, w);
            s_idx[0] = idx[0];
            s_idx[1] = idx[1];
            s_w[0] = w[0];
            s_w[1] = w[1];
            s_ramp = tidal_ramp(t, T.at_ramp);
        }
        __syncthreads();
    }
    const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= (LISTED ? lp.n : T.K) * P.nn) return;
    const int64_t e = item / P.nn;
    const int64_t k = LISTED ? (int64_t)lp.list[e] : e;
    const int64_t g = k * P.nn + item % P.nn;
    const int64_t nv = T.K * P.nn;
    double su = 0.0, sv = 0.0;
    const double h = in.h[g];
    if (!fp::lt(h, T.at_h_min)) {
        int idx[2];
        double w[2];
        int len;
        double ramp;
        if (LISTED) {
            const double t = lts_stage(lp, k).time;
            len = weather_weights(T.at_times, T.at_n_times, T.at_epoch + t, idx, w);
            ramp = tidal_ramp(t, T.at_ramp);
        } else {
            len = s_len;
            idx[0] = s_idx[0];
            idx[1] = s_idx[1];
            w[0] = s_w[0];
            w[1] = s_w[1];
            ramp = s_ramp;
        }
        const double rw = T.at_wind ? ramp : 0.0, rp = T.at_pressure ? ramp : 0.0;
        const double u = weather_field(T.at_values, nv, 0, g, idx, w, len);
        const double v = weather_field(T.at_values, nv, 1, g, idx, w, len);
        const double px = weather_field(T.at_values, nv, 2, g, idx, w, len);
        const double py = weather_field(T.at_values, nv, 3, g, idx, w, len);
        atmosphere_source(h, rw * u, rw * v, rp * px, rp * py, T.at_drag, T.at_cd, T.at_rho_air,
                          T.at_rho_water, T.at_h_min, su, sv);
    }
    if (T.rx_n > 0) T.rx_src[g] = 0.0;
    T.rx_src[nv + g] = su;
    T.rx_src[2 * nv + g] = sv;
}

// The weather's inverse-barometer level at flat node g and simulation time
// t (GriddedAtmosphere2D's BoundaryLevel by node index,
// gridded_atmosphere.rs:873-895), 0 unless the level is the pressure's
__device__ __forceinline__ double weather_level(const DevTables& T, const Physics& P, int64_t g,
                                                double t) {
    if (!T.at_level) return 0.0;
    int idx[2];
    double w[2];
    const int len = weather_weights(T.at_times, T.at_n_times, T.at_epoch + t, idx, w);
    const double p = weather_field(T.at_values, T.K * P.nn, 4, g, idx, w, len);
    return inverse_barometer_level(p, tidal_ramp(t, T.at_ramp), T.at_rho_water);
}

// A thread a face node. In FP64 the pipe was full (86 % of it; 0.348 ms for
// 200,000 quads at N = 3); in fixed point the integer pipes and the FP64
// pipe (the rotations, the conversions, faces that fixed point leaves) share
// the work at 59 to 64 % each and 0.106 ms. Four blocks an SM (64 registers, 112
// to 148 bytes spilled) against three or two: 10.48, 10.72, 11.16 ms over 60
// passes.
// LISTED: a multirate pass's faces (lp's edge and boundary-face lists),
// each boundary face at its element's stage time
template <int N1, bool LISTED>
__global__ void __launch_bounds__(256, DGSWE_FAST ? 4 : 2)
    face_kernel(DevTables T, Physics P, DevBuf in, double* fb_h, double* fb_hu, double* fb_hv,
                const StepCtl* ctl, int slot, const int* active, LtsPass lp) {
    if (!*active) return;
    const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n_int = (LISTED ? lp.n_edges : T.n_edges) * N1;
    if (item >= n_int + (LISTED ? lp.n_bfaces : T.n_bfaces) * N1) return;
    constexpr int NN = N1 * N1;
    const double g = P.g, h_min = P.h_min, sqrt_g = P.sqrt_g, half_g = P.half_g;
    if (item < n_int) {
        const int64_t e = LISTED ? (int64_t)lp.edges[item / N1] : item / N1;
        const int fi = (int)(item % N1);
        const int64_t L = T.edge_left[e], R = T.edge_right[e];
        const int64_t kl = L >> 2, kr = R >> 2;
        const int fl = (int)(L & 3), fr = (int)(R & 3);
        const int rfi = N1 - 1 - fi;
        const int nl = P.face_node[fl][fi], nr = P.face_node[fr][rfi];
        const int64_t gl = kl * NN + nl, gr = kr * NN + nr;
        F3 fa, fbb;
        if (P.formulation == kWetDry) {
            const Sd ql = load_side(in, T, P, gl), qr = load_side(in, T, P, gr);
            const double* geo = &T.edge_geo[e * 5];
#if DGSWE_FAST
            const FacePair f = face_pair(T, ql, qr, geo, g, sqrt_g, half_g, h_min);
#else
            const FacePair f = face_hll(ql, qr, geo, g, sqrt_g, half_g, h_min);
#endif
            fa = f.a;
            fbb = {fp::neg(f.b.h), fp::neg(f.b.hu), fp::neg(f.b.hv)};
        } else {
            const double* geo = &T.edge_geo[e * 5];
            entropy_surface(load_q(in, T, P, gl), load_q(in, T, P, gr), geo[0], geo[1], P, fa,
                            fbb);
        }
        const int64_t sl = (L * N1) + fi, sr = (R * N1) + rfi;
        fb_h[sl] = fa.h;
        fb_hu[sl] = fa.hu;
        fb_hv[sl] = fa.hv;
        fb_h[sr] = fbb.h;
        fb_hu[sr] = fbb.hu;
        fb_hv[sr] = fbb.hv;
        return;
    }
    // boundary face node (src/solver/rhs/swe_2d_split_form.rs:1090-1123)
    const int64_t bfi = LISTED ? (int64_t)lp.bfaces[(item - n_int) / N1] : (item - n_int) / N1;
    const int fi = (int)((item - n_int) % N1);
    const int64_t B = T.bface[bfi];
    const int64_t k = B >> 2;
    const int face = (int)(B & 3);
    const int node = P.face_node[face][fi];
    const Q qi = load_q(in, T, P, k * NN + node);
    const double* geo = &T.bface_geo[bfi * 5];
    const double nx = geo[0], ny = geo[1];
    const Condition& c = T.cond[T.bface_cond[bfi]];
    F3 fs;
    double u, v;
    interior_velocity(qi, h_min, u, v);
    if (c.kind == kBcWall) {
        const Q qe = wall_ghost(qi, u, v, nx, ny, c.wall_h_min, h_min);
        F3 fdummy;
        if (P.formulation == kWetDry)
#if DGSWE_FAST
            fs = face_pair(T, side(qi), side(qe), geo, g, sqrt_g, half_g, h_min).a;
#else
            fs = face_hll(side(qi), side(qe), geo, g, sqrt_g, half_g, h_min).a;
#endif
        else
            entropy_surface(qi, qe, nx, ny, P, fs, fdummy);
    } else {
        // CharacteristicOBC, flux F(q_b)·n: a uniform harmonic tide, or the
        // tide per boundary node (characteristic_boundary_state,
        // src/boundary/characteristic.rs:411-437)
        const int member = T.elem_member ? T.elem_member[k] : 0;
        // a multirate pass: the element's own stage time; a listed global
        // pass (no levels): the stage's
        const double t =
            (LISTED && lp.level) ? lts_stage(lp, k).time : ctl[member].stage[slot].time;
        Q qb;
        if (c.kind == kBcNodeTides || c.kind == kBcParent) {
            const int64_t s = T.bface_slot[bfi * N1 + fi];
            double eta, ue, ve;
            bool has_uv;
            if (c.kind == kBcNodeTides)
                node_tide_state(T.nt_omega + c.nt_omega0, T.nt_frate + c.nt_omega0,
                                T.nt_coef + c.nt_coef0 + (s - c.nt_slot0) * c.nt_n * 6, c.nt_n, t,
                                c.ramp, c.nt_use_mean ? T.nt_mean[s] : 0.0, c.nt_velocity,
                                c.nt_max_ratio, T.nt_depth[s], qi.b, eta, ue, ve, has_uv);
            else
                parent_state_at(T.pt_times + c.pt_time0, c.pt_n_times, c.pt_cubic,
                                T.pt_values + c.pt_val0 + (s - c.nt_slot0) * c.pt_n_times * 3, t,
                                c.ramp, c.pt_reference_level, c.nt_velocity, c.nt_max_ratio,
                                T.nt_depth[s], qi.b, eta, ue, ve, has_uv);
            if (c.raise) eta += c.raise_factor * weather_level(T, P, k * NN + node, t);
            const double h_e = fmax(eta - qi.b, 0.0);
            double un_e = 0.0, ut_e;
            if (has_uv) {
                un_e = ue * nx + ve * ny;
                ut_e = -ue * ny + ve * nx;
            } else {
                if (c.elevation_only == kIncomingWave)
                    un_e = 2.0 * (vsqrt(g * fmax(-qi.b, 0.0)) - vsqrt(g * h_e));
                ut_e = -u * ny + v * nx;
            }
            qb = characteristic_state_ext(qi, h_e, un_e, ut_e, nx, ny, g, h_min);
        } else {
            double eta = tide_elevation(c, t);
            if (c.raise) eta += c.raise_factor * weather_level(T, P, k * NN + node, t);
            qb = characteristic_state(qi, u, v, eta, nx, ny, c.elevation_only, g, h_min);
        }
        fs = wflux(qb, qb, nx, ny, g);
    }
    const int64_t sl = B * N1 + fi;
    fb_h[sl] = fs.h;
    fb_hu[sl] = fs.hu;
    fb_hv[sl] = fs.hv;
}

// ---------------------------------------------------------------------------
// the stage kernel

// SHAPE 0: ⌊128/NN⌋ elements a block; SHAPE 1: ⌊64/NN⌋ elements a block
// at twice the blocks per SM (the same registers and warps per SM); SHAPE 2:
// ⌊128/NN⌋ elements a block at 6 blocks per SM. The launch shapes
// dgswe_autotune chooses between.
template <int N1, int SHAPE = 0>
struct Cfg {
    static constexpr int NN = N1 * N1;
    static constexpr int NP = N1 - 1;      // pairs a node owns
    static constexpr int NA = 2 * (N1 - 1);  // pairs a node is in
    static constexpr int PER = SHAPE == 1 ? 64 : 128;
    static constexpr int EPB = (PER / NN) > 0 ? (PER / NN) : 1;
    static constexpr int THREADS = EPB * NN;
    // stage_kernel blocks per SM. In fixed point the integer and FP64 pipes
    // are each about half busy and the rest is latency: 28 warps an SM (72
    // registers) against 20 (96) take the 200,000-quad N = 3 right-hand side
    // from 0.226 to 0.210 ms, N = 4 at 100,000 from 0.354 to 0.310. At 72
    // registers orders 2 and 4 spill 24 and 16 bytes, 1 and 3 none; against 24
    // warps (80 registers) N = 1 to 4 take 76, 164, 174, 244 µs and 80, 168, 183,
    // 244 (400,000, 300,000, 200,000, 100,000 quads). The exact
    // numerics wait on the FP64 pipe: 20 warps (≤ 102 registers, no spills)
    // were 5 % faster than 16.
    static constexpr int MIN_BLOCKS =
        SHAPE == 2 ? 6 : (DGSWE_FAST ? 7 : 5) * (SHAPE == 1 ? 2 : 1);
    static constexpr int PAIR_DOUBLES = NN * NP * 3;
    static constexpr int FACE_DOUBLES = 2 * NN * 8;           // reconstructed faces
    static constexpr int NSUB = 2 * N1 * (N1 - 1);            // subcell interfaces
    static constexpr int IFL_DOUBLES = NSUB * 6;               // their fluxes
    // An element's scratch in FP64: its nodes' six values, and behind them the
    // pair fluxes or the subcells' reconstructed faces. The interface fluxes
    // come when the nodes' values are done with and lie over them.
    static constexpr int NODES = 6 * NN;
    static constexpr int AFTER = NODES > IFL_DOUBLES ? NODES : IFL_DOUBLES;
    static constexpr int X =
        AFTER + (PAIR_DOUBLES > FACE_DOUBLES ? PAIR_DOUBLES : FACE_DOUBLES);
    // In fixed point: the pair fluxes, the nodes' numbers, the lifted fluxes
    static constexpr int XF = PAIR_DOUBLES + 5 * NN + 12 * N1;
};

// LANES lanes work on an element; where that is a power of two they share a
// warp, and the element's exchanges through shared memory order that warp alone
template <int LANES>
constexpr bool kElementInWarp = LANES <= 32 && (LANES & (LANES - 1)) == 0;

template <int LANES>
__device__ __forceinline__ void element_sync() {
    if (kElementInWarp<LANES>) __syncwarp();
    else __syncthreads();
}

// Asks for the line at p to be in the L2 cache by the time it is read
__device__ __forceinline__ void prefetch(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// general_kernel: two lanes a node
template <int N1>
struct GenCfg {
    static constexpr int LANES = 2 * N1 * N1;
    static constexpr int EPB = 128 / LANES > 0 ? 128 / LANES : 1;
    static constexpr int THREADS = EPB * LANES;
    // Where an element's lanes straddle warps (N1 = 3), a warp waits for the
    // branches of up to three; as few elements as two a sub-partition have a
    // warp each instead (the block's last, two lanes short, holds one too): a
    // 4,000-quad drying channel's run 89.0 → 82.7 ms, a 50,000-quad box's the
    // same. At N1 = 2, where four fit a warp, that was 2 % slower (a
    // 90,000-quad storm, 129.9 → 132.7 ms).
    static constexpr bool SPREAD = LANES < 32 && 32 % LANES != 0;
    static constexpr unsigned FEW = 2 * 4 * 152;
};

__device__ __forceinline__ int line_node(int n1, int dir, int line, int pos) {
    return dir == 0 ? line * n1 + pos : pos * n1 + line;
}

// The subcell interface directions of one line (src/solver/rhs/subcells.rs:63-92)
template <int N1>
__device__ void telescoped(const Physics& P, const double (&m0)[N1], const double (&m1)[N1],
                           bool affine, double (&i0)[N1 + 1], double (&i1)[N1 + 1]) {
    if (affine) {
#pragma unroll
        for (int a = 0; a <= N1; ++a) {
            i0[a] = m0[0];
            i1[a] = m1[0];
        }
        return;
    }
    i0[0] = m0[0];
    i1[0] = m1[0];
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int a = 0; a < N1 - 1; ++a) {
#pragma unroll
        for (int c = 0; c < N1; ++c) {
            if (c == a) continue;
            const double q2 = 2.0 * P.w[a] * P.d[a * N1 + c];
            s0 += q2 * 0.5 * (m0[a] + m0[c]);
            s1 += q2 * 0.5 * (m1[a] + m1[c]);
        }
        i0[a + 1] = s0;
        i1[a + 1] = s1;
    }
    i0[N1] = m0[N1 - 1];
    i1[N1] = m1[N1 - 1];
}

template <int N1>
__device__ __forceinline__ void line_metric(const DevTables& T, int64_t k, int dir, int line,
                                            double (&m0)[N1], double (&m1)[N1]) {
    constexpr int NN = N1 * N1;
#pragma unroll
    for (int p = 0; p < N1; ++p) {
        const int64_t g = k * NN + line_node(N1, dir, line, p);
        m0[p] = T.contra[g * 4 + 2 * dir];
        m1[p] = T.contra[g * 4 + 2 * dir + 1];
    }
}

__device__ __forceinline__ int max_expo(double x, double y) {
    return max(fx::expo(x), fx::expo(y));
}

// The subcell interfaces' metrics of every element, [K][2·N1·(N1−1)][2] in
// the order of the subcell mass fluxes: what `telescoped` sums (72 FP64
// operations a direction at N = 3, twice per node of a subcell element)
template <int N1>
__global__ void __launch_bounds__(256) sub_metric_kernel(DevTables T, Physics P, double* out) {
    constexpr int NSUB = 2 * N1 * (N1 - 1);
    const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= T.K * 2 * N1) return;
    const int64_t k = item / (2 * N1);
    const int dir = (int)(item % (2 * N1)) / N1, line = (int)(item % N1);
    double m0[N1], m1[N1], i0[N1 + 1], i1[N1 + 1];
    line_metric<N1>(T, k, dir, line, m0, m1);
    telescoped<N1>(P, m0, m1, T.affine[k] != 0, i0, i1);
    double* o = &out[(k * NSUB + (dir * N1 + line) * (N1 - 1)) * 2];
#pragma unroll
    for (int pos = 0; pos + 1 < N1; ++pos) {
        o[2 * pos] = i0[pos + 1];
        o[2 * pos + 1] = i1[pos + 1];
    }
}

// The metric at end `at` of a line's subcells: of the interfaces, and of the
// line's end nodes (0, N1)
template <int N1>
__device__ __forceinline__ double subcell_metric(const DevTables& T, int64_t k, int dir, int line,
                                                 int at, int c) {
    if (at > 0 && at < N1)
        return T.sub_metric[2 * ((k * 2 + dir) * N1 * (N1 - 1) + line * (N1 - 1) + at - 1) + c];
    const int n = line_node(N1, dir, line, at == 0 ? 0 : N1 - 1);
    return T.contra[(k * N1 * N1 + n) * 4 + 2 * dir + c];
}

// The two slots of an element's face fluxes that a node takes, in the
// reference's face order, −1: none. A node lies on at most one s-face (0 or
// 2) and one r-face (1 or 3).
template <int N1>
__device__ __forceinline__ void node_slots(int a, int j, int& s_a, int& s_b) {
    int f_a = j == 0 ? 0 : (j == N1 - 1 ? 2 : -1);
    int f_b = a == N1 - 1 ? 1 : (a == 0 ? 3 : -1);
    if (f_a == 2 && f_b == 1) {
        f_a = 1;
        f_b = 2;
    }
    auto slot = [&](int f) {
        return f * N1 + (f == 0 ? a : (f == 1 ? j : (f == 2 ? N1 - 1 - a : N1 - 1 - j)));
    };
    s_a = f_a >= 0 ? slot(f_a) : -1;
    s_b = f_b >= 0 ? slot(f_b) : -1;
}

// −LIFT·sJ·F* of the node's faces added to its volume term r, over J. Every
// lane takes two slots, a missing one as zero, so the warp's instructions run
// on all lanes instead of once per face with only that face's nodes active.
// Subtracting +0 is exact.
template <int N1>
__device__ __forceinline__ F3 lift_only(const DevTables& T, const double* fb_h,
                                        const double* fb_hu, const double* fb_hv, int64_t k, int i,
                                        F3 r) {
    double c_a = 0.0, h_a = 0.0, hu_a = 0.0, hv_a = 0.0;
    double c_b = 0.0, h_b = 0.0, hu_b = 0.0, hv_b = 0.0;
    const int64_t fbase = k * 4 * N1;
    int s_a, s_b;
    node_slots<N1>(i % N1, i / N1, s_a, s_b);
    if (s_a >= 0) {
        c_a = T.lift_scale[fbase + s_a];
        h_a = fb_h[fbase + s_a];
        hu_a = fb_hu[fbase + s_a];
        hv_a = fb_hv[fbase + s_a];
    }
    if (s_b >= 0) {
        c_b = T.lift_scale[fbase + s_b];
        h_b = fb_h[fbase + s_b];
        hu_b = fb_hu[fbase + s_b];
        hv_b = fb_hv[fbase + s_b];
    }
    r.h -= c_a * h_a;
    r.hu -= c_a * hu_a;
    r.hv -= c_a * hv_a;
    r.h -= c_b * h_b;
    r.hu -= c_b * hu_b;
    r.hv -= c_b * hv_b;
    const double jinv = T.jinv[k * N1 * N1 + i];
    return {jinv * r.h, jinv * r.hu, jinv * r.hv};
}

// A node's right-hand side by the FP64 formulas, before the sources: an
// element with subcells (sub; dry: without water at any node), or a wet one.
// s_x is the element's scratch and holds its nodes' h, hu, hv, u, v and bed.
// SPLIT 2: two lanes a node (`half` 0 and 1), a direction of the subcells
// each; the result is the first's. Every lane of the element, or of the block
// where elements cross warps, calls it (take: the element takes part).
template <int N1, int SPLIT>
__device__ __forceinline__ F3 general_rhs(const DevTables& T, const Physics& P,
                                          const StageExtra& X, const DevBuf& in,
                                          const double* fb_h, const double* fb_hu,
                                          const double* fb_hv, int64_t k, int i, int half,
                                          bool take, bool sub, bool dry, double* s_x) {
    using C = Cfg<N1>;
    constexpr int NN = C::NN, NP = C::NP, NA = C::NA, LANES = SPLIT * NN;
    double(*const s_q)[NN] = (double(*)[NN])s_x;
    double* const pairs = s_x + C::AFTER;
    const bool wet = take && !sub && half == 0;
    const int a = i % N1, j = i / N1;
    const int64_t gi = k * NN + i;
    const double g = P.g, h_min = P.h_min, sqrt_g = P.sqrt_g, half_g = P.half_g;
    double h = 0.0, b = 0.0;
    if (take) {
        h = s_q[0][i];
        b = s_q[5][i];
    }
    double rh = 0.0, rhu = 0.0, rhv = 0.0;
    const bool affine = take ? T.affine[k] != 0 : true;

    auto node_side = [&](int n) { return Sd{s_q[0][n], s_q[3][n], s_q[4][n], s_q[5][n]}; };
    double* const faces = s_x + C::AFTER;  // [dir][line][pos][8]
    double* const ifl = s_x;               // [dir][line][pos][6]

    // ---- phase A: pair fluxes, or the subcells' reconstructed faces ----
    if (wet) {
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const int8_t* own = &T.sched_owned[(i * NP + q) * 5];
            const int na = own[0], nc = own[1];
            const double hm0 = T.pair_hm[(gi * NP + q) * 2];
            const double hm1 = T.pair_hm[(gi * NP + q) * 2 + 1];
            const double hc = s_q[0][nc];
            // ½·F#(q_a, q_c)·{{Ja}} scaled: mass, 2·F_hu, 2·F_hv
            const double mass = (s_q[1][na] + s_q[1][nc]) * hm0 +
                                (s_q[2][na] + s_q[2][nc]) * hm1;
            const double gp2 = P.two_g * s_q[0][na] * hc;
            const double g_hu = mass * (s_q[3][na] + s_q[3][nc]) + gp2 * hm0;
            const double g_hv = mass * (s_q[4][na] + s_q[4][nc]) + gp2 * hm1;
            double* slot_f = &pairs[(i * NP + q) * 3];
            slot_f[0] = mass;
            slot_f[1] = g_hu;
            slot_f[2] = g_hv;
        }
    } else if (take && sub && !dry) {
        // subcell faces of this node's subcell on its r-line and s-line
#pragma unroll 1
        for (int dir = half; dir < 2; dir += SPLIT) {
            const int line = dir == 0 ? j : a;
            const int pos = dir == 0 ? a : j;
            const Sd q = node_side(i);
            Sd l{}, r{};
            double x_l = 0.0, x_r = 0.0;
            bool have_l = true, have_r = true;
            if (pos > 0) {
                l = node_side(line_node(N1, dir, line, pos - 1));
                x_l = P.x[pos - 1];
            } else {
                // r-lines end on faces 3 (reversed) and 1; s-lines on 0 and 2 (reversed)
                const int face = dir == 0 ? 3 : 0;
                const int fi = dir == 0 ? N1 - 1 - line : line;
                const int64_t o = (k * 4 + face) * N1 + fi;
                const int64_t og = T.outer_idx[o];
                have_l = og >= 0;
                if (have_l) {
                    l = Sd{in.h[og], in.u[og], in.v[og], P.has_bed ? T.bed[og] : 0.0};
                    x_l = -1.0 - T.outer_dist[o];
                }
            }
            if (pos + 1 < N1) {
                r = node_side(line_node(N1, dir, line, pos + 1));
                x_r = P.x[pos + 1];
            } else {
                const int face = dir == 0 ? 1 : 2;
                const int fi = dir == 0 ? line : N1 - 1 - line;
                const int64_t o = (k * 4 + face) * N1 + fi;
                const int64_t og = T.outer_idx[o];
                have_r = og >= 0;
                if (have_r) {
                    r = Sd{in.h[og], in.u[og], in.v[og], P.has_bed ? T.bed[og] : 0.0};
                    x_r = 1.0 + T.outer_dist[o];
                }
            }
            Sd fl = q, fr = q;
            if (have_l && have_r)
                reconstruct(l, q, r, x_l, P.x[pos], x_r, X.xl[pos], X.xr[pos], P.subcell_h_dry,
                            fl, fr);
            double* f = &faces[((dir * N1 + line) * N1 + pos) * 8];
            f[0] = fl.h;
            f[1] = fl.u;
            f[2] = fl.v;
            f[3] = fl.b;
            f[4] = fr.h;
            f[5] = fr.u;
            f[6] = fr.v;
            f[7] = fr.b;
        }
    }
    element_sync<LANES>();

    // ---- phase B: sum the pairs; or the subcell interface fluxes ----
    if (wet) {
#pragma unroll
        for (int q = 0; q < NA; ++q) {
            const int slot_id = T.sched_slot[i * NA + q];
            const double coef = T.sched_coef[i * NA + q];
            const double hcoef = T.sched_hcoef[i * NA + q];  // coef / 2
            const double* f = &pairs[slot_id * 3];
            rh -= coef * f[0];
            rhu -= hcoef * f[1];
            rhv -= hcoef * f[2];
        }
        if (P.has_bed) {
            rhu -= h * T.gdb[gi * 2];
            rhv -= h * T.gdb[gi * 2 + 1];
        }
    } else if (take && dry) {
        if (X.subcell_mass)  // the dry element's interface fluxes are ±0
            for (int q = i + half * NN; q < C::NSUB; q += LANES)
                X.subcell_mass[k * C::NSUB + q] = 0.0;
    } else if (take && sub && !dry) {
#pragma unroll 1
        for (int dir = half; dir < 2; dir += SPLIT) {
            const int line = dir == 0 ? j : a;
            const int pos = dir == 0 ? a : j;
            if (pos + 1 >= N1) continue;
            const int64_t at = k * C::NSUB + (dir * N1 + line) * (N1 - 1) + pos;
            const double mx = subcell_metric<N1>(T, k, dir, line, pos + 1, 0);
            const double my = subcell_metric<N1>(T, k, dir, line, pos + 1, 1);
            const double norm = vsqrt(mx * mx + my * my);
            const double inv = vrcp(norm);
            const double geo[5] = {mx, my, norm, mx * inv, my * inv};
            const double* fa_ = &faces[((dir * N1 + line) * N1 + pos) * 8 + 4];   // right face of pos
            const double* fb_ = &faces[((dir * N1 + line) * N1 + pos + 1) * 8];   // left face of pos+1
            const Sd qa{fa_[0], fa_[1], fa_[2], fa_[3]}, qb{fb_[0], fb_[1], fb_[2], fb_[3]};
#if DGSWE_FAST
            const FacePair f = face_pair(T, qa, qb, geo, g, sqrt_g, half_g, h_min);
#else
            const FacePair f = face_hll(qa, qb, geo, g, sqrt_g, half_g, h_min);
#endif
            const F3 fa = f.a, fb = f.b;
            double* o = &ifl[((dir * N1 + line) * (N1 - 1) + pos) * 6];
            if (X.subcell_mass)  // subcell_slot (src/solver/rhs/subcells.rs:37-42)
                X.subcell_mass[at] = fa.h;
            o[0] = fa.h;
            o[1] = fa.hu;
            o[2] = fa.hv;
            o[3] = fb.h;
            o[4] = fb.hu;
            o[5] = fb.hv;
        }
    }
    element_sync<LANES>();

    // ---- phase C: the subcells' fluxes and bed terms at this node ----
    if (take && sub && !dry) {
#pragma unroll 1
        for (int dir = half; dir < 2; dir += SPLIT) {
            const int line = dir == 0 ? j : a;
            const int pos = dir == 0 ? a : j;
            const double iw = X.inv_w[pos];
            if (pos + 1 < N1) {
                const double* o = &ifl[((dir * N1 + line) * (N1 - 1) + pos) * 6];
                rh -= iw * o[0];
                rhu -= iw * o[1];
                rhv -= iw * o[2];
            }
            if (pos > 0) {
                const double* o = &ifl[((dir * N1 + line) * (N1 - 1) + pos - 1) * 6];
                rh += iw * o[3];
                rhu += iw * o[4];
                rhv += iw * o[5];
            }
            const double* f = &faces[((dir * N1 + line) * N1 + pos) * 8];
            const double lh = f[0], lb = f[3], rhh = f[4], rb = f[7];
            const double w_a = P.w[pos];
#if DGSWE_FAST
            (void)w_a;
            const double bed = -0.5 * g * (lh + rhh) * (rb - lb) * iw;  // iw = 1/w_a
#else
            const double bed = -0.5 * g * (lh + rhh) * (rb - lb) / w_a;
#endif
            double fx, fy;
            if (affine) {
                fx = bed * subcell_metric<N1>(T, k, dir, line, 0, 0);
                fy = bed * subcell_metric<N1>(T, k, dir, line, 0, 1);
            } else {
                const double ml0 = subcell_metric<N1>(T, k, dir, line, pos, 0);
                const double ml1 = subcell_metric<N1>(T, k, dir, line, pos, 1);
                const double mr0 = subcell_metric<N1>(T, k, dir, line, pos + 1, 0);
                const double mr1 = subcell_metric<N1>(T, k, dir, line, pos + 1, 1);
                const double metric =
#if DGSWE_FAST
                    0.25 * g * ((rhh + h) * (b - rb) + (lh + h) * (b - lb)) * iw;
#else
                    0.25 * g * ((rhh + h) * (b - rb) + (lh + h) * (b - lb)) / w_a;
#endif
                fx = bed * 0.5 * (ml0 + mr0) + metric * (mr0 - ml0);
                fy = bed * 0.5 * (ml1 + mr1) + metric * (mr1 - ml1);
            }
            rhu += fx;
            rhv += fy;
        }
    }

    if (SPLIT == 2) {  // the second direction's sums to the node's first lane
        element_sync<LANES>();  // the faces are done with
        if (half == 1) {
            faces[3 * i] = rh;
            faces[3 * i + 1] = rhu;
            faces[3 * i + 2] = rhv;
        }
        element_sync<LANES>();
        if (half == 0 && !wet) {
            rh += faces[3 * i];
            rhu += faces[3 * i + 1];
            rhv += faces[3 * i + 2];
        }
    }

    if (!take || half != 0) return {0.0, 0.0, 0.0};
    return lift_only<N1>(T, fb_h, fb_hu, fb_hv, k, i, F3{rh, rhu, rhv});
}

#if DGSWE_FAST
// A node's pair and lift terms of the mass by the FP64 formulas, for a slow node
// of an element in fixed point (a few in a thousand; listing the element for
// general_kernel instead made its launch behind every stage 6 µs longer). A call,
// out of the stage kernel's code and registers: 4.23 ms a step in it for a 1 M-quad
// box, 4.38 inlined
template <int N1>
__device__ __noinline__ double mass_sum(const DevTables& T, const DevBuf& in,
                                           const double* fb_h, uint64_t slots, int64_t k, int i,
                                           int s_a, int s_b) {
    constexpr int NN = N1 * N1, NP = N1 - 1, NA = 2 * NP;
    const double hu = in.hu[k * NN + i], hv = in.hv[k * NN + i];
    double r = 0.0;
#pragma unroll 2
    for (int q = 0; q < NA; ++q) {
        const int slot = (int)((slots >> (8 * q)) & 0xFF), owner = slot / NP;
        const int other = (T.fx_node[owner].others >> (8 * (slot - owner * NP))) & 0xFF;
        const int64_t o = k * NN + (owner == i ? other : owner);
        const double* hm = &T.pair_hm[(k * NN * NP + slot) * 2];
        r -= T.sched_coef[i * NA + q] * ((hu + in.hu[o]) * hm[0] + (hv + in.hv[o]) * hm[1]);
    }
    const int64_t fbase = k * 4 * N1;
    if (s_a >= 0) r -= T.lift_scale[fbase + s_a] * fb_h[fbase + s_a];
    if (s_b >= 0) r -= T.lift_scale[fbase + s_b] * fb_h[fbase + s_b];
    return r;
}

// Two a word: the depth's key (a negative depth's sign with it, which no scale
// takes) and 65535 less it, the same of the momentum, the exponent fields of the
// velocity and of the face fluxes' mass and momentum. Their maxima over an
// element's nodes and face slots give the element's fx::Exps.
struct ExpWords {
    unsigned w[4];
};

__device__ __forceinline__ unsigned both_ends(unsigned key) { return key | (65535u - key) << 16; }

__device__ __forceinline__ ExpWords node_exponents(double h, double hu, double hv, double u,
                                                   double v) {
    const unsigned m = max(fx::key(hu) & 0x7FFF, fx::key(hv) & 0x7FFF);
    return {{both_ends((unsigned)fx::key(h)), both_ends(m), (unsigned)max_expo(u, v), 0u}};
}

// The maxima over each NN lanes of a warp
template <int NN>
__device__ __forceinline__ void warp_max(ExpWords& e) {
#pragma unroll
    for (int off = NN / 2; off > 0; off >>= 1)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            e.w[q] = __vmaxu2(e.w[q], __shfl_xor_sync(0xffffffffu, e.w[q], off));
}

// The depths' part of an element's exponents from their keys' maxima
__device__ __forceinline__ fx::Exps depth_exponents(unsigned w) {
    fx::Exps x{};
    const int deepest = (int)(w & 0xFFFFu);
    x.h_key = 65535 - (int)(w >> 16);
    x.h_max = deepest >> 4;
    x.h_min = x.h_key >> 4;
    x.h_top = deepest & 15;
    return x;
}

__device__ __forceinline__ fx::Exps exponents(const ExpWords& e) {
    fx::Exps x = depth_exponents(e.w[0]);
    x.m = (int)(e.w[1] & 0xFFFFu) >> 4;
    x.m_key = 65535 - (int)(e.w[1] >> 16);
    x.v = (int)e.w[2];
    x.fh = (int)(e.w[3] & 0xFFFFu);
    x.fm = (int)(e.w[3] >> 16);
    return x;
}

// Of 2g, the 64ths above it and its key (fx::scales)
__device__ __forceinline__ int two_g_64ths(const DevTables& T) { return (T.fx_two_g.hi >> 24) + 1; }

// Whether an element's depths alone take it to FP64 (fx::thin_depth)
__device__ __forceinline__ bool thin_depth(const DevTables& T, const Physics& P, const FxExp& t,
                                           const fx::Exps& x) {
    return t.ok != 0 && fx::thin_depth(x, t, T.fx_e2g, two_g_64ths(T), fx::key(P.two_g));
}

// The fixed-point tables of each element from its FP64 ones: a warp per
// element takes the largest exponents, then cuts the entries to them
template <int N1>
__global__ void __launch_bounds__(256) fixed_tables_kernel(DevTables T, FxPair* hm, FxPair* gdb,
                                                           FxLimb* lift, FxExp* exps) {
    constexpr int NN = N1 * N1, NH = NN * (N1 - 1), NL = 4 * N1, NA = 2 * (N1 - 1);
    const int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (k >= T.K) return;
    const double* m = &T.pair_hm[k * NH * 2];
    const double* b = T.gdb ? &T.gdb[k * NN * 2] : nullptr;
    const double* l = &T.lift_scale[k * NL];
    int et = 0, eg = 0, el = 0;
    for (int q = lane; q < NH * 2; q += 32) et = max(et, fx::expo(m[q]));
    for (int q = lane; b && q < NN * 2; q += 32) eg = max(eg, fx::expo(b[q]));
    for (int q = lane; q < NL; q += 32) el = max(el, fx::expo(l[q]));
    et = __reduce_max_sync(0xffffffffu, et);
    eg = __reduce_max_sync(0xffffffffu, eg);
    el = __reduce_max_sync(0xffffffffu, el);
    fx::OwnMetric own{0x7FFF, 0x7FFF};
    for (int n = lane; n < NN; n += 32) {
        const fx::OwnMetric o = fx::own_metric(m, &T.sched_slot[n * NA], &T.sched_coef[n * NA], NA);
        own = {min(own.w, o.w), min(own.v, o.v)};
    }
    own = {__reduce_min_sync(0xffffffffu, own.w), __reduce_min_sync(0xffffffffu, own.v)};
    const bool ok = et >= fx::kExpLo && et <= fx::kExpHi && el >= fx::kExpLo && el <= fx::kExpHi &&
                    eg <= fx::kExpHi;
    eg = max(eg, fx::kExpLo - 400);  // a flat bed: no slope to scale by
    auto pair = [](double x, double y, int K) {
        return FxPair{fx::split(fx::to_fixed(x, K)), fx::split(fx::to_fixed(y, K))};
    };
    for (int q = lane; q < NH; q += 32)
        hm[k * NH + q] = pair(m[2 * q], m[2 * q + 1], et + 1);
    for (int q = lane; q < NN; q += 32)
        gdb[k * NN + q] = b ? pair(b[2 * q], b[2 * q + 1], eg + 1) : FxPair{};
    for (int q = lane; q < NL; q += 32) lift[k * NL + q] = fx::split(fx::to_fixed(l[q], el + 2));
    if (lane == 0)
        exps[k] = {et - 1022, eg - 1022, el - 1022,
                   ok ? fx::own_deficits(own, et - 1022, T.fx_ec) : 0};
}
#endif

// A node's stage from its right-hand side F: the sources, the combination,
// the damping, then the accumulation or the wet/dry correction and the
// output. LANES lanes an element, of which the first NN hold its nodes
// (valid); s_q is scratch of the element's, s_flag and s_red its own.
template <int N1, bool LISTED, int LANES>
__device__ __forceinline__ void finish_node(const DevTables& T, const Physics& P,
                                            const DevBuf& in, const DevBuf& base,
                                            const DevBuf& out, const DevBuf& acc,
                                            const DevBuf& keep, StepCtl* cm, const LtsPass& lp,
                                            int slot, int mode, int check_finite, int64_t k, int i,
                                            bool valid, const F3& F, double (*s_q)[N1 * N1],
                                            int* s_flag, double* s_red) {
    constexpr int NN = N1 * N1;
    const int tid = threadIdx.x;
    const int64_t gi = k * NN + i;
    const double h_min = P.h_min;
    // read (again, from the cache: ten registers fewer until here)
    double h = 0.0, hu = 0.0, hv = 0.0, u = 0.0, v = 0.0;
    if (valid) {
        h = in.h[gi];
        hu = in.hu[gi];
        hv = in.hv[gi];
        u = in.u[gi];
        v = in.v[gi];
    }
    // ---- the sources ----
    double Fh = F.h, Fhu = F.hu, Fhv = F.hv;
    if (valid) {
        if (P.has_coriolis) {
            const double f = P.coriolis_field ? T.fcor[gi] : P.f0;
            Fhu += f * hv;
            Fhv += -f * hu;
        }
        if (T.rx_src) {  // the nesting relaxation band (0 off the band)
            const int64_t nv = T.K * NN;
            Fh += T.rx_src[gi];
            Fhu += T.rx_src[nv + gi];
            Fhv += T.rx_src[2 * nv + gi];
        }
        if (mode == kRhsOnly) {
            out.h[gi] = Fh;
            out.hu[gi] = Fhu;
            out.hv[gi] = Fhv;
        }
    }
    if (mode == kRhsOnly) return;  // uniform: no barrier follows for this mode

    // ---- stage combination and damping ----
    const StageArgs sa = LISTED ? (valid ? lts_stage(lp, k) : StageArgs{}) : cm->stage[slot];
    double vh = 0.0, vhu = 0.0, vhv = 0.0;
    if (valid) {
        if (fp::bits(sa.a) == 0x3FF0000000000000ll) {  // 1: no multiply
            vh = base.h[gi];
            vhu = base.hu[gi];
            vhv = base.hv[gi];
        } else if (fp::nz(sa.a)) {
            vh = sa.a * base.h[gi];
            vhu = sa.a * base.hu[gi];
            vhv = sa.a * base.hv[gi];
        }
        if (fp::nz(sa.b)) {
            vh += sa.b * h;
            vhu += sa.b * hu;
            vhv += sa.b * hv;
        }
        if (fp::nz(sa.c)) {
            vh += sa.c * Fh;
            vhu += sa.c * Fhu;
            vhv += sa.c * Fhv;
        }
        // for the adjoint: the combination, then the damped momentum
        if (keep.h) {
            keep.h[gi] = vh;
            keep.hu[gi] = vhu;
            keep.hv[gi] = vhv;
        }
        if (P.friction || P.has_wet_dry) {
            const double g_n2 = P.friction == 2 ? T.g_n2[gi] : P.g_n2;
            damp(P, g_n2, vh, vhu, vhv, DampIn{h, hu, hv, u, v}, sa.c);
        }
        if (keep.h) {
            keep.u[gi] = vhu;
            keep.v[gi] = vhv;
        }
    }

    if (mode == kAccumulate) {
        if (valid) {
            out.h[gi] = vh;
            out.hu[gi] = vhu;
            out.hv[gi] = vhv;
            const double w = sa.w, keep = sa.keep;
            if (fp::nz(keep)) {
                acc.h[gi] = w * vh + keep * acc.h[gi];
                acc.hu[gi] = w * vhu + keep * acc.hu[gi];
                acc.hv[gi] = w * vhv + keep * acc.hv[gi];
            } else {
                acc.h[gi] = w * vh;
                acc.hu[gi] = w * vhu;
                acc.hv[gi] = w * vhv;
            }
        }
        return;
    }

    // ---- wet/dry correction (wetting_drying.rs:194-215) ----
    if (P.has_wet_dry) {
        const bool thin = valid && fp::lt(vh, P.h_dry);
        bool needs, some;  // the element's, and some element's of the group
        if (kElementInWarp<LANES>) {
            const unsigned lanes = (unsigned)(((1ull << LANES) - 1) << ((tid & 31) / LANES * LANES));
            const unsigned votes = __ballot_sync(0xffffffffu, thin);
            needs = (votes & lanes) != 0;
            some = votes != 0;
            __syncwarp();  // the element's scratch is free again
        } else {
            if (i == 0 && valid) *s_flag = 0;
            __syncthreads();
            if (thin) atomicOr(&*s_flag, 1);
            some = __syncthreads_or(thin) != 0;
            needs = *s_flag != 0;
        }
        if (some) {
            if (valid) {
                s_q[0][i] = vh;
                s_q[1][i] = vhu;
                s_q[2][i] = vhv;
            }
            element_sync<LANES>();
        }
        if (valid && needs && i < 4) {
            // element_mean and positivity_limit_element
            // (src/solver/limiters/swe_2d.rs:135-203), in node order: a lane
            // for each mean, one for the smallest depth
            if (i < 3) {
                const double* mass = &T.mass[k * NN];
                double sum = 0.0;
#pragma unroll
                for (int p = 0; p < NN; ++p) sum += mass[p] * s_q[i][p];
                s_red[i] = sum * T.inv_area[k];
                if (i == 0 && fp::lt0(s_red[0]))
                    atomicAdd((unsigned long long*)&cm->clips, 1ull);
            } else {
                double hmin = INFINITY;
                for (int p = 0; p < NN; ++p) hmin = lmin(s_q[0][p], hmin);
                s_red[3] = hmin;
            }
        }
        if (some) element_sync<LANES>();
        if (valid && needs) {
            const double h_avg = s_red[0];
            if (fp::le0(h_avg)) {
                vh = vhu = vhv = 0.0;
            } else {
                const double hmin = s_red[3];
                if (fp::lt0(hmin)) {
                    double th = vdiv(h_avg, h_avg - hmin);
                    th = fp::lt0(th) ? 0.0 : (fp::gt(th, 1.0) ? 1.0 : th);
                    vh = th * (vh - h_avg) + h_avg;
                    vhu = th * (vhu - s_red[1]) + s_red[1];
                    vhv = th * (vhv - s_red[2]) + s_red[2];
                    vh = fp::max0(vh);
                }
                if (fp::lt(h_avg, P.h_dry)) vhu = vhv = 0.0;
            }
        }
        if (valid) correct_node(P, vh, vhu, vhv);
    }
    if (valid) {
        out.h[gi] = vh;
        out.hu[gi] = vhu;
        out.hv[gi] = vhv;
        double uo, vo;
        node_velocity(vh, vhu, vhv, h_min, uo, vo);
        out.u[gi] = uo;
        out.v[gi] = vo;
        if (check_finite && !(fp::finite(vh) && fp::finite(vhu) && fp::finite(vhv)))
            cm->nonfinite = 1;
    }
}

#if DGSWE_FAST
// The wet elements of a stage in fixed point, and those without water at any
// node, which only their faces' fluxes reach (their reconstructed subcell
// faces are dry, so the interface fluxes, pressure and bed terms are all ±0).
// Any other with subcells, and one that fixed point leaves to FP64 (fixed64.hpp),
// goes into T.gen_list's second half for general_kernel, launched behind
// (shallow_listed: those with subcells, and those left by their depths, are in its
// first half already, and a
// general_kernel takes them beside this kernel): inside this kernel its few hundred FP64
// operations in a row (a call, so spills on the wet path; one busy warp to a
// block's end) cost 17 % of a 50,000-quad coastal box's stage.
// LISTED: a multirate pass over lp's elements, each with its own stage
template <int N1, bool LISTED, int SHAPE = 0>
__global__ void __launch_bounds__(Cfg<N1, SHAPE>::THREADS, Cfg<N1, SHAPE>::MIN_BLOCKS)
    stage_kernel(const __grid_constant__ DevTables T, Physics P, StageExtra X,
                 const __grid_constant__ DevBuf in, DevBuf base, DevBuf out, DevBuf acc,
                 const double* __restrict__ fb_h, const double* __restrict__ fb_hu,
                 const double* __restrict__ fb_hv, StepCtl* ctl, int slot, int mode,
                 int check_finite, const int* active, DevBuf keep, LtsPass lp,
                 int shallow_listed) {
    using C = Cfg<N1, SHAPE>;
    constexpr int NN = C::NN, NP = C::NP, NA = C::NA, EPB = C::EPB;
    // an element whose lanes share a warp finds its flags and largest
    // exponents by votes and shuffles, else in shared memory
    constexpr bool kInWarp = kElementInWarp<NN>;
    __shared__ double s_x[EPB][C::XF];
    __shared__ int s_flag[EPB][3];
    __shared__ double s_red[EPB][4];
    __shared__ unsigned s_exp[kInWarp ? 1 : EPB][8];

    const int run = *active;
    const int tid = threadIdx.x;
    const int e = tid / NN, i = tid % NN;
    int64_t k = (int64_t)blockIdx.x * EPB + e;
    if (LISTED) k = k < lp.n ? (int64_t)lp.list[k] : T.K;
    else k += X.k_first;
    const int64_t k_end = (LISTED || X.k_last > T.K) ? T.K : X.k_last;
    // the element's member (its StepCtl); an ensemble member that has
    // stopped keeps its state: its elements take no part
    StepCtl* const cm = ctl + ((T.elem_member && k < k_end) ? T.elem_member[k] : 0);
    const bool valid = k < k_end && (!T.elem_member || cm->active);
    const int64_t gi = k * NN + i;
    const int64_t fbase = k * 4 * N1;  // the element's face slots
    double(*const s_q)[NN] = (double(*)[NN])s_x[e];

    // the node, and the element's 4·N1 face slots dealt out to its nodes
    constexpr int NS = (4 * N1 + NN - 1) / NN;
    double h = 0, hu = 0, hv = 0, u = 0, v = 0, flux[NS][3];
    if (valid) {
        h = in.h[gi];
        hu = in.hu[gi];
        hv = in.hv[gi];
        u = in.u[gi];
        v = in.v[gi];
    }
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        const int sl = i + q * NN;
        const bool has = valid && sl < 4 * N1;
        flux[q][0] = has ? fb_h[fbase + sl] : 0.0;
        flux[q][1] = has ? fb_hu[fbase + sl] : 0.0;
        flux[q][2] = has ? fb_hv[fbase + sl] : 0.0;
    }
    if (valid) {
        // what the later phases read, on its way from DRAM meanwhile
        prefetch(&T.fx_hm[gi * NP]);
        prefetch(&T.fx_gdb[gi]);
        prefetch(&T.jinv[gi]);
        prefetch(&T.fx_lift[fbase + i % (4 * N1)]);
        prefetch(&T.fx_exp[k]);
    }
    if (!run) return;
    ExpWords ew = node_exponents(h, hu, hv, u, v);
#pragma unroll
    for (int q = 0; q < NS; ++q)
        ew.w[3] = __vmaxu2(ew.w[3], (unsigned)(fx::expo(flux[q][0]) |
                                               max_expo(flux[q][1], flux[q][2]) << 16));
    const bool shallow = valid && P.formulation == kWetDry && fp::lt(h, P.subcell_depth);
    // sub: the element has a node below the subcell depth; dry: no water at any
    bool sub, dry;
    if (kInWarp) {
        const unsigned lanes = (unsigned)(((1ull << NN) - 1) << ((tid & 31) / NN * NN));
        sub = (__ballot_sync(0xffffffffu, shallow) & lanes) != 0;
        dry = (__ballot_sync(0xffffffffu, shallow && !fp::nz(h)) & lanes) == lanes;
        warp_max<NN>(ew);
    } else {
        if (i < 2) s_flag[e][i] = 0;
        for (int q = i; q < 8; q += NN) s_exp[e][q] = 0;
        __syncthreads();
        if (shallow) {
            atomicOr(&s_flag[e][0], 1);
            if (!fp::nz(h)) atomicAdd(&s_flag[e][1], 1);
        }
        for (int q = 0; q < 4; ++q) {
            atomicMax(&s_exp[e][2 * q], ew.w[q] & 0xFFFFu);
            if (q != 2) atomicMax(&s_exp[e][2 * q + 1], ew.w[q] >> 16);
        }
        __syncthreads();
        sub = s_flag[e][0] != 0;
        dry = s_flag[e][1] == NN;
        for (int q = 0; q < 4; ++q) ew.w[q] = s_exp[e][2 * q] | s_exp[e][2 * q + 1] << 16;
    }
    // fixed: the element's right-hand side comes from here; slow: the mass of a
    // node may not
    bool fixed = false, slow = false;
    fx::Scale sc;
    if (valid && !sub) {
        const FxExp t = T.fx_exp[k];
        const fx::Exps x = exponents(ew);
        sc = fx::scales(x, t, T.fx_ec, T.fx_e2g, two_g_64ths(T));
        fixed = sc.ok && !fx::thin(x, sc, t, fx::key(P.two_g));
        slow = fixed && fx::slow_node(x, sc, t, T.fx_e2g);
        if (slow) prefetch(&T.pair_hm[gi * NP * 2]);
    }
    if (valid && !fixed && !dry && i == 0) {
        const bool listed =
            shallow_listed && (sub || (P.formulation == kWetDry &&
                                       thin_depth(T, P, T.fx_exp[k], depth_exponents(ew.w[0]))));
        if (!listed) T.gen_list[T.K + atomicAdd(&T.gen_count[2], 1u)] = (int32_t)k;
    }

    FxLimb G{}, H{};                         // 2g·h, h
    int64_t m0 = 0, m1 = 0, u0 = 0, u1 = 0;  // hu, hv, u, v
    FxLimb* const pairs = (FxLimb*)&s_x[e][0];
    FxLimb* const nd_h = (FxLimb*)&s_x[e][C::PAIR_DOUBLES];
    int64_t* const nd = (int64_t*)&s_x[e][C::PAIR_DOUBLES + NN];
    int64_t* const lifted = (int64_t*)&s_x[e][C::PAIR_DOUBLES + 5 * NN];
    if (fixed) {
        H = fx::split(fx::to_fixed_nn(h, sc.kh));
        G = fx::two_g_h(H, T.fx_two_g, sc);
        m0 = fx::to_fixed(hu, sc.km);
        m1 = fx::to_fixed(hv, sc.km);
        u0 = fx::to_fixed(u, sc.ku);
        u1 = fx::to_fixed(v, sc.ku);
        nd_h[i] = H;
        nd[i] = m0;
        nd[NN + i] = m1;
        nd[2 * NN + i] = u0;
        nd[3 * NN + i] = u1;
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            const int sl = i + q * NN;
            if (sl >= 4 * N1) continue;
            const FxLimb c = T.fx_lift[fbase + sl];
            lifted[sl] = fx::mul<0>(c, fx::split(fx::to_fixed(flux[q][0], sc.kfh)));
            lifted[4 * N1 + sl] = fx::mul<0>(c, fx::split(fx::to_fixed(flux[q][1], sc.kfm)));
            lifted[8 * N1 + sl] = fx::mul<0>(c, fx::split(fx::to_fixed(flux[q][2], sc.kfm)));
        }
    }
    const FxNode node = T.fx_node[i];
    element_sync<NN>();

    // ---- the pair fluxes ----
    if (fixed) {
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const int o = (node.others >> (8 * q)) & 0xFF;  // the pair's other node
            const FxPair hm = T.fx_hm[gi * NP + q];
            const fx::Flux f = fx::pair_flux(G, nd_h[o], m0 + nd[o], m1 + nd[NN + o],
                                             u0 + nd[2 * NN + o], u1 + nd[3 * NN + o], hm.x, hm.y);
            FxLimb* slot_f = &pairs[(i * NP + q) * 3];
            slot_f[0] = f.h;
            slot_f[1] = f.hu;
            slot_f[2] = f.hv;
        }
    }
    element_sync<NN>();

    // ---- their sums, the bed slope, the lift and 1/J ----
    F3 F{0.0, 0.0, 0.0};
    if (fixed) {
        fx::PairSum ah = fx::pair_sum(), au = ah, av = ah;
#pragma unroll
        for (int q = 0; q < NA; ++q) {
            const FxLimb* f = &pairs[(int)((node.slots >> (8 * q)) & 0xFF) * 3];
            const FxLimb coef = T.fx_coef[i * NA + q];
            fx::mac(ah, coef, f[0]);
            fx::mac(au, coef, f[1]);
            fx::mac(av, coef, f[2]);
        }
        int64_t fh = -fx::fold(ah), fhu = -fx::fold(au), fhv = -fx::fold(av);
        if (P.has_bed) {
            const FxPair slope = T.fx_gdb[gi];
            fhu -= fx::bed_term(H, slope.x, sc);
            fhv -= fx::bed_term(H, slope.y, sc);
        }
        int s_a, s_b;
        node_slots<N1>(i % N1, i / N1, s_a, s_b);
        for (const int sl : {s_a, s_b})
            if (sl >= 0) {
                fh -= lifted[sl];
                fhu -= lifted[4 * N1 + sl];
                fhv -= lifted[8 * N1 + sl];
            }
        const double jinv = T.jinv[gi];
        F.h = fx::over_jacobian(fh, sc.sh, jinv);
        if (slow) {  // a node whose own mass terms are too small takes them in FP64
            int64_t own = 0;
#pragma unroll
            for (int q = 0; q < NA; ++q)
                fx::own_mass(own, T.fx_coef[i * NA + q],
                             pairs[(int)((node.slots >> (8 * q)) & 0xFF) * 3]);
            if (s_a >= 0) fx::own_mass(own, lifted[s_a]);
            if (s_b >= 0) fx::own_mass(own, lifted[s_b]);
            if (fx::own_mass_small(own))
                F.h = jinv * mass_sum<N1>(T, in, fb_h, node.slots, k, i, s_a, s_b);
        }
        F.hu = fx::over_jacobian(fhu, sc.sm, jinv);
        F.hv = fx::over_jacobian(fhv, sc.sm, jinv);
        if (X.subcell_mass)  // no subcells: NaN (compute_rhs_swe_2d_mass_fluxes_into)
            for (int q = i; q < C::NSUB; q += NN)
                X.subcell_mass[k * C::NSUB + q] = fp::from_bits(0x7FF8000000000000ll);
    }
    if (dry) {
        F = lift_only<N1>(T, fb_h, fb_hu, fb_hv, k, i, F3{0.0, 0.0, 0.0});
        if (X.subcell_mass)  // its interface fluxes are ±0
            for (int q = i; q < C::NSUB; q += NN) X.subcell_mass[k * C::NSUB + q] = 0.0;
    }
    // the buffer summed into may be the input, which a slow node's mass_sum reads
    // at the element's other nodes
    if (mode == kAccumulate) element_sync<NN>();
    finish_node<N1, LISTED, NN>(T, P, in, base, out, acc, keep, cm, lp, slot, mode, check_finite, k,
                                i, fixed || dry, F, s_q, &s_flag[e][2], s_red[e]);
}

// A stage's elements with subcells and water and those whose depths leave them
// to FP64, from its input, into T.gen_list's first half: beside the face pass, so
// that general_kernel can take them beside the stage pass
template <int N1>
__global__ void __launch_bounds__(256)
    shallow_list_kernel(DevTables T, Physics P, DevBuf in, const StepCtl* ctl,
                        const int* active) {
    constexpr int NN = N1 * N1, EPB = 256 / NN;
    __shared__ int s_flag[EPB][2];
    __shared__ unsigned s_key[EPB][2];
    if (!*active) return;
    const int e = threadIdx.x / NN, i = threadIdx.x % NN;
    const int64_t k = (int64_t)blockIdx.x * EPB + e;
    const bool valid = e < EPB && k < T.K && (!T.elem_member || ctl[T.elem_member[k]].active);
    const double h = valid ? in.h[k * NN + i] : 0.0;
    const bool shallow = valid && fp::lt(h, P.subcell_depth);
    unsigned ends = both_ends((unsigned)fx::key(h));
    bool sub, dry;
    if (kElementInWarp<NN>) {
        const unsigned lanes = (unsigned)(((1ull << NN) - 1) << ((threadIdx.x & 31) / NN * NN));
        sub = (__ballot_sync(0xffffffffu, shallow) & lanes) != 0;
        dry = (__ballot_sync(0xffffffffu, shallow && !fp::nz(h)) & lanes) == lanes;
#pragma unroll
        for (int off = NN / 2; off > 0; off >>= 1)
            ends = __vmaxu2(ends, __shfl_xor_sync(0xffffffffu, ends, off));
    } else {
        if (e < EPB && i < 2) s_flag[e][i] = 0, s_key[e][i] = 0;
        __syncthreads();
        if (e < EPB) {
            atomicMax(&s_key[e][0], ends & 0xFFFFu);
            atomicMax(&s_key[e][1], ends >> 16);
        }
        if (shallow) {
            atomicOr(&s_flag[e][0], 1);
            if (!fp::nz(h)) atomicAdd(&s_flag[e][1], 1);
        }
        __syncthreads();
        if (e >= EPB) return;
        sub = s_flag[e][0] != 0;
        dry = s_flag[e][1] == NN;
        ends = s_key[e][0] | s_key[e][1] << 16;
    }
    if (valid && i == 0 && (sub ? !dry : thin_depth(T, P, T.fx_exp[k], depth_exponents(ends))))
        T.gen_list[atomicAdd(&T.gen_count[0], 1u)] = (int32_t)k;
}

// The elements of a stage that stage_kernel leaves (a half of T.gen_list):
// those with subcells, and wet ones that FP64 is closer to. Few and long
// (some 200 FP64 operations in a row, 20 µs for any number of them), so two
// lanes a node, a subcell direction each. The last block to end empties the
// list for the next stage.
template <int N1, bool LISTED>
__global__ void __launch_bounds__(GenCfg<N1>::THREADS, 4)
    general_kernel(const __grid_constant__ DevTables T, const __grid_constant__ Physics P,
                   const __grid_constant__ StageExtra X, const __grid_constant__ DevBuf in,
                   DevBuf base, DevBuf out, DevBuf acc, const double* __restrict__ fb_h,
                   const double* __restrict__ fb_hu, const double* __restrict__ fb_hv, StepCtl* ctl,
                   int slot, int mode, int check_finite, const int* active, DevBuf keep,
                   LtsPass lp, int list) {
    constexpr int NN = N1 * N1, LANES = 2 * NN, EPB = GenCfg<N1>::EPB;
    using C = Cfg<N1>;
    __shared__ double s_x[EPB][C::X];
    __shared__ int s_flag[EPB][2];
    __shared__ double s_red[EPB][4];
    const int tid = threadIdx.x;
    const int32_t* elements = T.gen_list + list * T.K;
    unsigned* const count = T.gen_count + 2 * list;
    const unsigned n = *active ? *(volatile unsigned*)count : 0u;
    // where they are few, a warp each
    constexpr int WARPS = (GenCfg<N1>::THREADS + 31) / 32;
    const bool spread = GenCfg<N1>::SPREAD && n <= GenCfg<N1>::FEW && n <= gridDim.x * WARPS;
    const int stride = spread ? 32 : LANES;
    const unsigned per_block = spread ? WARPS : EPB;
    const int e = tid / stride, lane = tid % stride, half = lane / NN, i = lane % NN;
    double(*const s_q)[NN] = (double(*)[NN])s_x[e];
    for (unsigned first = blockIdx.x * per_block; first < n; first += gridDim.x * per_block) {
        const bool listed = first + e < n && lane < LANES;
        const int64_t k = listed ? (int64_t)elements[first + e] : 0;
        StepCtl* const cm = ctl + ((T.elem_member && listed) ? T.elem_member[k] : 0);
        const bool take = listed && (!T.elem_member || cm->active);
        const int64_t gi = k * NN + i;
        double h = 0.0;
        if (take && half == 0) {
            h = in.h[gi];
            s_q[0][i] = h;
            s_q[1][i] = in.hu[gi];
            s_q[2][i] = in.hv[gi];
            s_q[3][i] = in.u[gi];
            s_q[4][i] = in.v[gi];
            s_q[5][i] = P.has_bed ? T.bed[gi] : 0.0;
        }
        // sub: an element with a node below the subcell depth
        const bool shallow =
            take && half == 0 && P.formulation == kWetDry && fp::lt(h, P.subcell_depth);
        if (lane == 0) s_flag[e][0] = 0;
        element_sync<LANES>();
        if (shallow) atomicOr(&s_flag[e][0], 1);
        element_sync<LANES>();
        const bool sub = s_flag[e][0] != 0;
        const F3 F = general_rhs<N1, 2>(T, P, X, in, fb_h, fb_hu, fb_hv, k, i, half, take, sub,
                                        false, s_x[e]);
        if (X.subcell_mass && take && !sub)  // no subcells: NaN
            for (int q = lane; q < C::NSUB; q += LANES)
                X.subcell_mass[k * C::NSUB + q] = fp::from_bits(0x7FF8000000000000ll);
        finish_node<N1, LISTED, LANES>(T, P, in, base, out, acc, keep, cm, lp, slot, mode,
                                       check_finite, k, i, take && half == 0, F, s_q,
                                       &s_flag[e][1], s_red[e]);
        element_sync<LANES>();
    }
    __syncthreads();
    if (tid == 0 && atomicAdd(&count[1], 1u) == gridDim.x - 1) {
        count[0] = 0;
        count[1] = 0;
    }
}
#else
// LISTED: a multirate pass over lp's elements, each with its own stage
template <int N1, bool LISTED, int SHAPE = 0>
__global__ void __launch_bounds__(Cfg<N1, SHAPE>::THREADS, Cfg<N1, SHAPE>::MIN_BLOCKS)
    stage_kernel(DevTables T, Physics P, StageExtra X, DevBuf in, DevBuf base, DevBuf out,
                 DevBuf acc, const double* __restrict__ fb_h, const double* __restrict__ fb_hu,
                 const double* __restrict__ fb_hv, StepCtl* ctl, int slot, int mode,
                 int check_finite, const int* active, DevBuf keep, LtsPass lp) {
    using C = Cfg<N1, SHAPE>;
    constexpr int NN = C::NN, EPB = C::EPB;
    __shared__ double s_x[EPB][C::X];
    __shared__ int s_flag[EPB][3];
    __shared__ double s_red[EPB][4];

    if (!*active) return;
    const int tid = threadIdx.x;
    const int e = tid / NN, i = tid % NN;
    int64_t k = (int64_t)blockIdx.x * EPB + e;
    if (LISTED) k = k < lp.n ? (int64_t)lp.list[k] : T.K;
    else k += X.k_first;
    const int64_t k_end = (LISTED || X.k_last > T.K) ? T.K : X.k_last;
    // the element's member (its StepCtl); an ensemble member that has
    // stopped keeps its state: its elements take no part
    StepCtl* const cm = ctl + ((T.elem_member && k < k_end) ? T.elem_member[k] : 0);
    const bool valid = k < k_end && (!T.elem_member || cm->active);
    const int64_t gi = k * NN + i;
    double(*const s_q)[NN] = (double(*)[NN])s_x[e];
    double h = 0.0;
    if (valid) {
        h = in.h[gi];
        s_q[0][i] = h;
        s_q[1][i] = in.hu[gi];
        s_q[2][i] = in.hv[gi];
        s_q[3][i] = in.u[gi];
        s_q[4][i] = in.v[gi];
        s_q[5][i] = P.has_bed ? T.bed[gi] : 0.0;
    }
    if (i < 2) s_flag[e][i] = 0;
    // sub: an element with a node below the subcell depth; dry: without water
    // at any node (every h = ±0, so every u = v = 0): its reconstructed subcell
    // faces are dry, so the interface fluxes, pressure and bed terms are all
    // ±0, and it skips the subcell phases
    const bool shallow = valid && P.formulation == kWetDry && fp::lt(h, P.subcell_depth);
    element_sync<NN>();
    if (shallow) {
        atomicOr(&s_flag[e][0], 1);
        if (!fp::nz(h)) atomicAdd(&s_flag[e][1], 1);
    }
    element_sync<NN>();
    const bool sub = s_flag[e][0] != 0, dry = s_flag[e][1] == NN;
    const F3 F =
        general_rhs<N1, 1>(T, P, X, in, fb_h, fb_hu, fb_hv, k, i, 0, valid, sub, dry, s_x[e]);
    if (X.subcell_mass && valid && !sub)  // no subcells: NaN (compute_rhs_swe_2d_mass_fluxes_into)
        for (int q = i; q < C::NSUB; q += NN)
            X.subcell_mass[k * C::NSUB + q] = fp::from_bits(0x7FF8000000000000ll);
    finish_node<N1, LISTED, NN>(T, P, in, base, out, acc, keep, cm, lp, slot, mode, check_finite, k,
                                i, valid, F, s_q, &s_flag[e][2], s_red[e]);
}
#endif

// finish_where over every element: state ← acc, then the wet/dry correction
// LISTED: the end of the substeps of lp's elements, and a non-finite
// result flagged in ctl
template <int N1, bool LISTED>
__global__ void __launch_bounds__(Cfg<N1>::THREADS)
    finish_kernel(DevTables T, Physics P, DevBuf acc, DevBuf state, StepCtl* ctl, LtsPass lp) {
    using C = Cfg<N1>;
    constexpr int NN = C::NN, EPB = C::EPB;
    __shared__ double s_v[EPB][3][NN];
    __shared__ int s_flag[EPB];
    __shared__ double s_red[EPB][4];
    const int tid = threadIdx.x;
    const int e = tid / NN, i = tid % NN;
    int64_t k = (int64_t)blockIdx.x * EPB + e;
    if (LISTED) k = k < lp.n ? (int64_t)lp.list[k] : T.K;
    const bool valid = k < T.K;
    const int64_t gi = k * NN + i;
    StepCtl* const cm = ctl + ((T.elem_member && valid) ? T.elem_member[k] : 0);  // the member's
    if (i == 0) s_flag[e] = 0;
    double vh = 0, vhu = 0, vhv = 0;
    if (valid) {
        vh = acc.h[gi];
        vhu = acc.hu[gi];
        vhv = acc.hv[gi];
    }
    s_v[e][0][i] = vh;
    s_v[e][1][i] = vhu;
    s_v[e][2][i] = vhv;
    __syncthreads();
    if (P.has_wet_dry) {
        if (valid && fp::lt(vh, P.h_dry)) atomicOr(&s_flag[e], 1);
        __syncthreads();
        const bool needs = s_flag[e] != 0;
        if (valid && needs && i < 4) {
            // element_mean and positivity_limit_element
            // (src/solver/limiters/swe_2d.rs:135-203), in node order: a lane
            // for each mean, one for the smallest depth
            if (i < 3) {
                const double* mass = &T.mass[k * NN];
                double sum = 0.0;
#pragma unroll
                for (int p = 0; p < NN; ++p) sum += mass[p] * s_v[e][i][p];
                s_red[e][i] = sum * T.inv_area[k];
                if (i == 0 && fp::lt0(s_red[e][0]))
                    atomicAdd((unsigned long long*)&cm->clips, 1ull);
            } else {
                double hmin = INFINITY;
                for (int p = 0; p < NN; ++p) hmin = lmin(s_v[e][0][p], hmin);
                s_red[e][3] = hmin;
            }
        }
        __syncthreads();
        if (valid && needs) {
            const double h_avg = s_red[e][0];
            if (fp::le0(h_avg)) {
                vh = vhu = vhv = 0.0;
            } else {
                const double hmin = s_red[e][3];
                if (fp::lt0(hmin)) {
                    double th = vdiv(h_avg, h_avg - hmin);
                    th = fp::lt0(th) ? 0.0 : (fp::gt(th, 1.0) ? 1.0 : th);
                    vh = th * (vh - h_avg) + h_avg;
                    vhu = th * (vhu - s_red[e][1]) + s_red[e][1];
                    vhv = th * (vhv - s_red[e][2]) + s_red[e][2];
                    vh = fp::max0(vh);
                }
                if (fp::lt(h_avg, P.h_dry)) vhu = vhv = 0.0;
            }
        }
        if (valid) correct_node(P, vh, vhu, vhv);
    }
    if (valid) {
        state.h[gi] = vh;
        state.hu[gi] = vhu;
        state.hv[gi] = vhv;
        double uo, vo;
        node_velocity(vh, vhu, vhv, P.h_min, uo, vo);
        state.u[gi] = uo;
        state.v[gi] = vo;
        if (LISTED && !(fp::finite(vh) && fp::finite(vhu) && fp::finite(vhv))) cm->nonfinite = 1;
    }
}

// Per element, whether every node is deeper than each of three depths
// (bits 0, 1, 2): the line-local test and the two depths of the coarse
// step's bound (SWEPhysics2D::line_local and coarse_step_bound,
// src/physics/builder.rs:560-632)
__global__ void depth_flags_kernel(const double* h, int64_t K, int nn, double d0, double d1,
                                   double d2, uint8_t* flags) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    bool a = true, b = true, c = true;
    for (int i = 0; i < nn; ++i) {
        const double x = h[k * nn + i];
        a = a && fp::gt(x, d0);
        b = b && fp::gt(x, d1);
        c = c && fp::gt(x, d2);
    }
    flags[k] = (uint8_t)((a ? 1 : 0) | (b ? 2 : 0) | (c ? 4 : 0));
}

// The point-implicit damping of a stage value over dt with the rates frozen
// at `from` (apply_implicit_damping_2d, src/solver/algorithms/
// wetting_drying.rs:376-389: damp_node at every node), then the stage's
// node velocities
__global__ void damping_kernel(DevTables T, Physics P, DevBuf stage, DevBuf from, double dt,
                               int64_t n) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const double h = stage.h[g];
    double hu = stage.hu[g], hv = stage.hv[g];
    const double g_n2 = P.friction == 2 ? T.g_n2[g] : P.g_n2;
    damp(P, g_n2, h, hu, hv, DampIn{from.h[g], from.hu[g], from.hv[g], from.u[g], from.v[g]},
         dt);
    stage.hu[g] = hu;
    stage.hv[g] = hv;
    double u, v;
    node_velocity(h, hu, hv, P.h_min, u, v);
    stage.u[g] = u;
    stage.v[g] = v;
}

// node velocities of a buffer (after an upload)
__global__ void velocity_kernel(DevBuf b, int64_t n, double h_min) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    double u, v;
    node_velocity(b.h[g], b.hu[g], b.hv[g], h_min, u, v);
    b.u[g] = u;
    b.v[g] = v;
}

// ---------------------------------------------------------------------------
// the time step (src/solver/rhs/swe_2d.rs:2072-2115, 1346-1367, 2165-2258)

// The dt pass. An element's step needs only the largest of its nodes' rates
// (its own nodes and the neighbours' face nodes, each with its own metric),
// so the rates are first taken in single precision — on the FP32 and
// integer pipes, which run 64 times faster than the FP64 pipe — with a bound
// on their error; only the rates that can still be the largest are then
// computed in FP64, by dense lanes from a list in shared memory, and their
// maximum is the exact one. One lane per element then takes the positivity
// sums in node order, the reference's order.
//
// node_rate_f32 (point.cuh) is within 2⁻²⁰·B of the FP64 rate, B its error
// scale; a node whose r₃₂ + δ·B is below the largest r₃₂ − δ·B of its
// element (δ = 2⁻¹⁶, sixteen times the bound) cannot hold the maximum.
template <int N1>
struct DtCfg {
    static constexpr int NN = N1 * N1;
    // elements per block, one lane of warp 0 each: 16, so that a dt block
    // (256 threads at N = 3, 40 registers) fits on an SM beside two blocks
    // of the face pass it runs with
    static constexpr int EPB = 16;
    static constexpr int THREADS = EPB * NN;
    static constexpr int PITCH = NN + 1;  // odd row pitch: lanes spread over the banks
    static constexpr int SLOTS = NN + 4 * N1;  // own nodes, then neighbours' face nodes
};

// The element's dt from its largest rate and its nodes' depths and mass
// weights (element_dt, swe_2d.rs:2072-2115, with PositivityBound::element_cfl
// and positivity_relaxation, swe_2d.rs:2220-2258)
__device__ __forceinline__ double element_dt(const DtParams& D, int order, double weight_ratio,
                                             double rmax, double water, double water_b,
                                             bool shallow) {
    double cfl = D.cfl;
    if (D.positivity) {
        // f64::min drops the NaN of 0/0
        const double ratio =
            fp::le0(water_b) ? weight_ratio : lmin(water / water_b, weight_ratio);
        const double rho = lmax(0.9 * ratio, 1.0);
        const double cap = shallow ? D.max_cfl_subcells : D.max_cfl;
        cfl = lmin(cfl, lmin(D.bound_cfl * rho, cap));
    }
    return fp::lt(rmax, 1e-14) ? INFINITY : cfl / ((2.0 * (double)order + 1.0) * rmax);
}

// Whether node p lies on the element's boundary
template <int N1>
__device__ __forceinline__ constexpr bool boundary_node(int p) {
    return p % N1 == 0 || p % N1 == N1 - 1 || p / N1 == 0 || p / N1 == N1 - 1;
}

// The water over the element's nodes and over its boundary nodes, in node
// order, every product and sum rounded on its own (two kernels take it and
// the step must have the same bits from both)
__device__ __forceinline__ void add_water(double wi, bool boundary, double& water,
                                          double& water_b) {
    water = __dadd_rn(water, wi);
    if (boundary) water_b = __dadd_rn(water_b, wi);
}

// Every element's step into dt_el, and the smallest
template <int N1>
__global__ void __launch_bounds__(DtCfg<N1>::THREADS)
    dt_kernel(DevTables T, Physics P, DevBuf q, DtParams D, double* dt_el, StepCtl* ctl,
              const int* active) {
    using C = DtCfg<N1>;
    constexpr int NN = C::NN, EPB = C::EPB, PITCH = C::PITCH, SLOTS = C::SLOTS;
    __shared__ int64_t s_k[EPB];                      // the block's elements
    __shared__ float s_r[EPB][SLOTS];                 // r₃₂, −1 for a dry node
    __shared__ float s_b[EPB][SLOTS];                 // δ·B
    __shared__ unsigned int s_lo[EPB];                // the element's largest r₃₂ − δ·B (bits)
    __shared__ unsigned long long s_rmax[EPB];        // its largest exact rate (bits)
    __shared__ short s_list[EPB * SLOTS];             // candidates: e·SLOTS + slot
    __shared__ int s_count;
    __shared__ double s_h[EPB * PITCH];
    __shared__ double s_mass[EPB * PITCH];
    if (!*active) return;
    const int tid = threadIdx.x;
    const int e = tid / NN, i = tid % NN;
    const int64_t k = (int64_t)blockIdx.x * EPB + e;
    if (i == 0) s_k[e] = k;
    const int64_t gi = k * NN + i;
    const double g = P.g, h_min = P.h_min;
    const float g32 = f32_trunc(g);
    constexpr float kDelta = 1.0f / 65536.0f;      // δ = 2⁻¹⁶
    constexpr float kFloor = 1e-30f;               // the sub-float-range terms
    if (tid < EPB) {
        s_lo[tid] = 0u;
        s_rmax[tid] = 0ull;  // +0: a dry node's rate
    }
    if (tid == 0) s_count = 0;
    double h = 0.0, mass = 0.0;
    // single-precision rates of the node and of the neighbour face nodes it takes
    auto slot_rate = [&](int slot, double hs, double us, double vs, const float* m) {
        float r = -1.0f, b = 0.0f;
        if (fp::gt(hs, h_min)) {
            node_rate_f32(hs, us, vs, m, g32, r, b);
            b = kDelta * b + kFloor;
        }
        s_r[e][slot] = r;
        s_b[e][slot] = b;
    };
    if (k < T.K) {
        h = q.h[gi];
        mass = T.mass[gi];
        slot_rate(i, h, q.u[gi], q.v[gi], &T.dtm32_own[gi * 6]);
        for (int it = i; it < 4 * N1; it += NN) {
            const int64_t o = k * 4 * N1 + it;
            const int64_t nb = T.nb_face_node[o];
            if (nb < 0) {
                s_r[e][NN + it] = -1.0f;
                s_b[e][NN + it] = 0.0f;
                continue;
            }
            slot_rate(NN + it, q.h[nb], q.u[nb], q.v[nb], &T.dtm32_face[o * 6]);
        }
    }
    s_h[e * PITCH + i] = h;
    s_mass[e * PITCH + i] = mass;
    __syncthreads();
    // the element's threshold: its largest r₃₂ − δ·B (non-negative floats
    // order as their bits)
    if (k < T.K) {
        for (int sl = i; sl < SLOTS; sl += NN) {
            const float r = s_r[e][sl];
            if (r >= 0.0f) atomicMax(&s_lo[e], __float_as_uint(fmaxf(r - s_b[e][sl], 0.0f)));
        }
    }
    __syncthreads();
    if (k < T.K) {
        const float lo = __uint_as_float(s_lo[e]);
        for (int sl = i; sl < SLOTS; sl += NN) {
            const float r = s_r[e][sl];
            if (r >= 0.0f && r + s_b[e][sl] >= lo)
                s_list[atomicAdd(&s_count, 1)] = (short)(e * SLOTS + sl);
        }
    }
    __syncthreads();
    // exact rates of the candidates, one per lane
    const int n_cand = s_count;
    for (int c = tid; c < n_cand; c += C::THREADS) {
        const int es = s_list[c];
        const int ce = es / SLOTS, sl = es % SLOTS;
        const int64_t kc = s_k[ce];
        int64_t node;
        const double* m;
        if (sl < NN) {
            node = kc * NN + sl;
            m = &T.dtm_own[node * 6];
        } else {
            const int64_t o = kc * 4 * N1 + (sl - NN);
            node = T.nb_face_node[o];
            m = &T.dtm_face[o * 6];
        }
        const double r = node_rate(q.h[node], q.u[node], q.v[node], m, g);
        atomicMax(&s_rmax[ce], (unsigned long long)fp::bits(r));  // r ≥ +0
    }
    __syncthreads();
    if (tid >= 32) return;  // warp 0: lane l < EPB finishes the block's element l
    const int64_t kl = tid < EPB ? s_k[tid] : T.K;
    unsigned long long dt_bits = 0x7FF0000000000000ull;  // +∞
    int member = -1;
    if (kl < T.K) {
        const double rmax = fp::from_bits((int64_t)s_rmax[tid]);
        double water = 0.0, water_b = 0.0;
        bool shallow = false;
        if (D.positivity)
#pragma unroll
            for (int p = 0; p < NN; ++p) {
                const double hp = s_h[tid * PITCH + p];
                shallow = shallow || fp::le(hp, D.shallow);
                add_water(__dmul_rn(s_mass[tid * PITCH + p], fp::max0(hp)), boundary_node<N1>(p),
                          water, water_b);
            }
        const double dt = element_dt(D, P.order, T.weight_ratio[kl], rmax, water, water_b, shallow);
        dt_el[kl] = dt;
        dt_bits = (unsigned long long)fp::bits(dt);
        member = T.elem_member ? T.elem_member[kl] : 0;
    }
    // Each member's smallest step over the warp, then one atomic per member
    // present: members are contiguous element ranges, so lane l gathers the
    // lanes above it while they share its member, and the first lane of each
    // run holds that run's minimum. dt ≥ 0, so its bits order as the values.
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long o = __shfl_down_sync(0xffffffffu, dt_bits, off);
        const int om = __shfl_down_sync(0xffffffffu, member, off);
        if (tid + off < 32 && om == member && o < dt_bits) dt_bits = o;
    }
    const int below = __shfl_up_sync(0xffffffffu, member, 1);
    if (member >= 0 && (tid == 0 || below != member)) atomicMin(&ctl[member].dt_bits, dt_bits);
}

// The smallest step alone, where no element's own is asked for: the same
// bits as dt_kernel's minimum. Every element's step is bracketed in single
// precision (its largest rate between max(r₃₂ ∓ δ·B), its water ratio within
// 2⁻¹⁶); the smallest upper end so far, of all blocks, is kept beside the
// smallest step, and only an element whose lower end is not above it is
// taken in FP64. A few hundred elements are, and what remains is memory: 112 B
// a node, read at 58 % of the DRAM's rate (0.062 ms for 200,000 quads at
// N = 3, where dt_kernel takes 0.146). An element has LANES lanes of one warp,
// each with at most a node and a face slot.
// LISTED: the elements list[0..n_list) (any order, any subset), else all
template <int N1>
struct DtLanes {
    static constexpr int LANES = N1 == 2 ? 8 : (N1 == 5 ? 32 : 16);
    static constexpr int EPB = 256 / LANES;
};

template <int N1, bool LISTED>
__global__ void __launch_bounds__(256)
    dt_min_kernel(DevTables T, Physics P, DevBuf q, DtParams D, StepCtl* ctl, const int* active,
                  const int32_t* list, int64_t n_list) {
    constexpr int NN = N1 * N1, LANES = DtLanes<N1>::LANES, EPB = DtLanes<N1>::EPB;
    if (!*active) return;
    const int lane = threadIdx.x % LANES;
    const int64_t at = (int64_t)blockIdx.x * EPB + threadIdx.x / LANES;
    const int64_t k = LISTED ? (at < n_list ? (int64_t)list[at] : T.K) : at;
    const bool mine = k < T.K;
    StepCtl* const cm = ctl + ((T.elem_member && mine) ? T.elem_member[k] : 0);
    constexpr float kDelta = 1.0f / 65536.0f, kFloor = 1e-30f;  // δ = 2⁻¹⁶, as dt_kernel's
    const float g32 = f32_trunc(P.g);
    const int64_t gi = k * NN + lane, o = k * 4 * N1 + lane;
    const bool node = mine && lane < NN, slot = mine && lane < 4 * N1;
    double h = 0.0, mass = 0.0, u = 0.0, v = 0.0;
    double hf = 0.0, uf = 0.0, vf = 0.0;
    float m[6], mf[6];
    const int64_t nb = slot ? T.nb_face_node[o] : -1;
    if (node) {
        h = q.h[gi];
        u = q.u[gi];
        v = q.v[gi];
        mass = T.mass[gi];
        const float2* t = (const float2*)&T.dtm32_own[gi * 6];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 x = t[c];
            m[2 * c] = x.x;
            m[2 * c + 1] = x.y;
        }
    }
    if (nb >= 0) {
        hf = q.h[nb];
        uf = q.u[nb];
        vf = q.v[nb];
        const float2* t = (const float2*)&T.dtm32_face[o * 6];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 x = t[c];
            mf[2 * c] = x.x;
            mf[2 * c + 1] = x.y;
        }
    }
    // the rates in single precision, −1 for a dry or missing node
    float r = -1.0f, b = 0.0f, rf = -1.0f, bf = 0.0f;
    if (node && fp::gt(h, P.h_min)) {
        node_rate_f32(h, u, v, m, g32, r, b);
        b = kDelta * b + kFloor;
    }
    if (nb >= 0 && fp::gt(hf, P.h_min)) {
        node_rate_f32(hf, uf, vf, mf, g32, rf, bf);
        bf = kDelta * bf + kFloor;
    }
    float lo = fmaxf(fmaxf(r - b, rf - bf), 0.0f), up = fmaxf(fmaxf(r + b, rf + bf), 0.0f);
    const bool edge = boundary_node<N1>(lane);
    const float w32 = node ? f32_trunc(mass) * f32_trunc(fp::max0(h)) : 0.0f;
    float water32 = w32, water_b32 = edge ? w32 : 0.0f;
    unsigned thin = node && fp::le(h, D.shallow) ? 1u : 0u;
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) {
        lo = fmaxf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
        up = fmaxf(up, __shfl_xor_sync(0xffffffffu, up, off));
        water32 += __shfl_xor_sync(0xffffffffu, water32, off);
        water_b32 += __shfl_xor_sync(0xffffffffu, water_b32, off);
        thin |= __shfl_xor_sync(0xffffffffu, thin, off);
    }
    // the step between its bounds; each factor's rounding is within 2⁻²⁰
    const double weight_ratio = mine ? T.weight_ratio[k] : 1.0;
    float cfl_lo = D.cfl32, cfl_up = D.cfl32;
    if (D.positivity) {
        constexpr float kRatio = 1.0f / 65536.0f;
        const float wr = f32_trunc(weight_ratio);
        const float cap = thin ? D.max_cfl_subcells32 : D.max_cfl32;
        // water that single precision flushes: any ratio from 0 to the weights'
        const bool some = water_b32 > 1e-30f;
        const float ratio = some ? fminf(water32 / water_b32, wr) : wr;
        const float rho_lo = some ? fmaxf(0.9f * ratio * (1.0f - kRatio), 1.0f) : 1.0f;
        const float rho_up = fmaxf(0.9f * ratio * (1.0f + kRatio), 1.0f);
        cfl_lo = fminf(cfl_lo, fminf(D.bound_cfl32 * rho_lo, cap));
        cfl_up = fminf(cfl_up, fminf(D.bound_cfl32 * rho_up, cap));
    }
    constexpr float kStep = 1.0f / 131072.0f;  // 2⁻¹⁷
    const float n21 = 2.0f * (float)P.order + 1.0f;
    const float dt_lo = up > 0.0f ? cfl_lo / (n21 * up) * (1.0f - kStep) : INFINITY;
    const float dt_up = lo > 1e-13f ? cfl_up / (n21 * lo) * (1.0f + kStep) : INFINITY;
    // the smallest upper end so far (the bits of floats ≥ 0 order as they do),
    // read once for the element: other blocks lower it meanwhile, and its lanes
    // have to agree on whether it is taken
    unsigned best = 0x7F800000u;  // +∞
    if (mine && lane == 0) {
        best = *(volatile unsigned*)&cm->dt_up;
        if (__float_as_uint(dt_up) < best) atomicMin(&cm->dt_up, __float_as_uint(dt_up));
        best = min(best, __float_as_uint(dt_up));
    }
    best = __shfl_sync(0xffffffffu, best, 0, LANES);
    const bool exact = mine && __float_as_uint(dt_lo) <= best;
    if (!__any_sync(0xffffffffu, exact)) return;
    unsigned long long rmax = 0ull;  // the bits of rates ≥ +0
    if (exact && r >= 0.0f && r + b >= lo)
        rmax = (unsigned long long)fp::bits(node_rate(h, u, v, &T.dtm_own[gi * 6], P.g));
    if (exact && rf >= 0.0f && rf + bf >= lo) {
        const unsigned long long x =
            (unsigned long long)fp::bits(node_rate(hf, uf, vf, &T.dtm_face[o * 6], P.g));
        rmax = x > rmax ? x : rmax;
    }
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xffffffffu, rmax, off);
        rmax = x > rmax ? x : rmax;
    }
    const double wi = __dmul_rn(mass, fp::max0(h));
    double water = 0.0, water_b = 0.0;
    if (D.positivity)
        for (int p = 0; p < NN; ++p)
            add_water(__shfl_sync(0xffffffffu, wi, p, LANES), boundary_node<N1>(p), water, water_b);
    if (exact && lane == 0) {
        const double dt = element_dt(D, P.order, weight_ratio, fp::from_bits((int64_t)rmax), water,
                                     water_b, thin != 0u);
        atomicMin(&cm->dt_bits, (unsigned long long)fp::bits(dt));
    }
}

// ---------------------------------------------------------------------------
// the run's clock on the device (Simulation::run_with_callback's loop body,
// src/simulation/runner.rs:355-450)

constexpr int kFailDtMin = 4, kFailMaxSteps = 5, kFailNonFinite = 3;

// Whether the step runs: no failure, time left before the target, steps left
__global__ void step_begin(StepCtl* ctl, int n) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    StepCtl* c = ctl + m;
    c->dt_bits = 0x7FF0000000000000ull;  // +∞
    c->dt_up = 0x7F800000u;
    bool run = c->failure == 0 && c->t < c->target;
    if (run && c->max_steps > 0 && c->steps >= c->max_steps) {
        c->failure = kFailMaxSteps;
        run = false;
    }
    c->active = run ? 1 : 0;
    // the first stage's time needs no dt (its offset is 0 in every scheme):
    // set here, a pass of the first stage can start beside the dt pass
    if (run && c->st_c[0] == 0.0) c->stage[0].time = c->t;
}

// dt from the element steps, capped, checked, fitted to land on the target;
// the stages' times and weights (element_stage, src/time/multirate.rs:169-200)
__global__ void step_dt(StepCtl* ctl, int n) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    StepCtl* c = ctl + m;
    if (!c->active) return;
    double dt = __longlong_as_double((long long)c->dt_bits);
    if (c->dt_max > 0.0) dt = fmin(dt, c->dt_max);
    if (c->dt_min > 0.0 && dt < c->dt_min) {
        c->failure = kFailDtMin;
        c->active = 0;
        c->dt = dt;
        return;
    }
    c->dt_min_used = fmin(c->dt_min_used, dt);
    c->dt_max_used = fmax(c->dt_max_used, dt);
    const bool landed = c->t + dt * (1.0 + 1e-9) >= c->target;
    if (landed) dt = c->target - c->t;
    c->landed = landed ? 1 : 0;
    c->dt = dt;
    for (int s = 0; s < c->scheme_stages; ++s) {
        StageArgs& a = c->stage[s];
        if (s > 0 || c->st_c[0] != 0.0)  // the first stage's time from step_begin
            a.time = __dadd_rn(c->t, __dmul_rn(c->st_c[s], dt));  // rounded apart, as the reference
        a.a = c->st_start[s];
        a.b = c->st_input[s];
        a.c = c->st_beta[s] * dt;
        a.w = 1.0;
        a.keep = 0.0;
    }
}

__global__ void step_end(StepCtl* ctl, int n) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    StepCtl* c = ctl + m;
    if (!c->active) return;
    c->t = c->landed ? c->target : c->t + c->dt;
    c->steps += 1;
    if (c->nonfinite) {
        c->failure = kFailNonFinite;
        c->active = 0;
    }
}

}  // namespace DGSWE_NS
}  // namespace dgswe
