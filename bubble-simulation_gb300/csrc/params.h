// Parameter blocks shared by the host driver and the CUDA kernels.
//
// LatticeParams mirrors the `SimParams` uniform (shaders/common.wgsl:25-58,
// host values src/gpu/sim.rs:613-644) minus the fields no kernel on this path
// reads (time, vis_gain, padding).  It is templated on the arithmetic type so
// the FP64 kernels get double constants (each widened exactly from the f32
// value the host derives, so both precisions solve the same problem).
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define BUBBLE_HD __host__ __device__ __forceinline__
#else
#define BUBBLE_HD inline
#endif

namespace bubble {

template <typename R>
struct alignas(4 * sizeof(R)) V4 {
    R x, y, z, w;
};
template <typename R>
struct alignas(2 * sizeof(R)) V2 {
    R x, y;
};

template <typename R>
struct LatticeParams {
    int32_t nx, ny, nz, _pad;
    R dx, inv_dx, eta, lambda;
    R phi_b, m2, delta, wall_width;
    R p_floor, e_floor, z_max, e_ref;
    // Perturbation form: the background subtracted from the stored energy
    // (e_bg = e_ref) and from the pressure (p_bg = e_bg / 3); both 0, and the
    // floors unshifted, for the other forms.
    R e_bg, p_bg;
    // Gamma-law equation of state: c_s^2 = Gamma - 1 and the offset e0 of
    // e = p / (Gamma - 1) + e0; both 0 for the bag model.  eos_k = 1 / c_s^2 + 1
    // (the enthalpy is eos_k p + e0) and eos_cs = c_s, for the fast arithmetic.
    R eos_c2, eos_e0, eos_k, eos_cs;
    // Thermal potential V(phi) + gamma/2 (T^2 - T_ref^2) phi^2 - A/3 (T - T_ref) phi^3:
    // th_k = a/3, th_g = gamma, th_h = A/3, th_a = A, th_lo = sqrt(3 gamma / (4 a))
    // (the physical branch is T >= th_lo |phi|), th_i2a = 1/(2a), the radiation
    // constant a, T_ref and th_ik = 1 / th_k (fast arithmetic); all 0 for the
    // other equations of state.
    R th_k, th_g, th_h, th_a, th_lo, th_i2a, a_rad, t_ref, th_ik;
};

// One SSP-RK3 stage: U_out = a0 U^n + a1 (U_in + dt L(U_in))
// (shaders/common.wgsl:60-68, src/gpu/sim.rs:133-135, 650-656).
template <typename R>
struct StageArgs {
    const V2<R> *field_n;
    const V4<R> *fluid_n;
    const V2<R> *field_in;
    const V4<R> *fluid_in;
    V2<R> *field_out;
    V4<R> *fluid_out;
    R a0, a1, dt;
    int32_t stage;  // 0, 1, 2; stage 0 has a0 == 0 and never reads U^n
    // Bounded waits of the stage kernel give up after 2^wait_shift SM cycles.
    // Test hook (bubble_ext_test_expire_stage_wait): when test_tx != 0, every
    // CTA staging planes through TMA arms its first plane's mbarrier for
    // test_tx bytes and issues no copy for it, so that wait expires.
    uint32_t test_tx = 0;
    int32_t wait_shift = 31;
};

// Result of the diagnostics reduction (shaders/reduce.wgsl:32-38), with FP64
// sums.
struct DiagResult {
    double sums[4];       // e_total, broken, kinetic, E
    uint32_t max_v_bits;  // bits of max |v| (non-negative f32)
    uint32_t nonfinite;   // count of blocks that saw a non-finite term
    uint64_t cells;
};

// What a diagnostics launch leaves in pinned host memory: its result and the
// status word of the bounded waits.
struct HostReport {
    DiagResult result;
    int32_t status;
};

// Tile shape of the fused stage kernel.
struct TileShape {
    int32_t tx, ty, lz;  // x, y tile (cells) and z chunk (planes)
    int32_t form = 0;    // BUBBLE_STAGE_FORM_* of 16 x 16 FP32 launches of the column kernel
    int32_t pair_lz = 0; // z chunk of the pair form where lz was not set by the caller; 0: lz
};

// The stage kernel's tiles are 16 x 16 (FP32 default: the least perimeter,
// so the least halo work, for 256 column threads) or 32 x ty (ty = 8, 4):
// the tile height selects the width.
constexpr int tile_x_for(int ty) { return ty == 16 ? 16 : 32; }

// Cost model of one stage launch of the 16 x 16 FP32 column kernel, in plane
// times of a CTA that shares its SM with one other.  The register form holds
// two CTAs per SM, the shared form three, each then 1.4x slower per plane;
// the busiest SM (ceil(CTAs / SMs) CTAs) runs them in rounds, a last round
// of one CTA at 0.65x and of two (shared form) at 0.8x of the full round's
// plane time; a chunk costs its planes plus 2 for its warm-up.  Fitted to
// about 150 measured (form, chunk) pairs from 32^3 to 512^3: the cheapest
// pick (chunks of 4 planes or more) is the fastest measured or within 0.6 %
// of it at every size.
inline double column_stage_cost(uint32_t nx, uint32_t ny, uint32_t nz, int lz, bool shared, int sms) {
    if (lz < 1) lz = 1;
    if (sms < 1) sms = 1;
    const long tiles = (long)((nx + 15) / 16) * (long)((ny + 15) / 16);
    const long chunks = ((long)nz + lz - 1) / lz;
    const long lz_eff = ((long)nz + chunks - 1) / chunks;
    const long k = shared ? 3 : 2;
    const double p = shared ? 1.4 : 1.0;
    const long m = (tiles * chunks + sms - 1) / sms;
    const long rounds = (m + k - 1) / k;
    const long last = m - (rounds - 1) * k;
    const double p_last = last == k ? p : (last == 1 ? 0.65 * p : 0.8 * p);
    return ((double)(rounds - 1) * p + p_last) * (double)(lz_eff + 2);
}

// Cost model of one FP64 stage launch, in plane times of a CTA.  The FP64 pipes
// bound it (two operations per clock and SM on GB300), so an SM's time is the
// sum of its CTAs' planes, each chunk costing 0.73 of a plane for its warm-up:
// 16 x 16 tiles measure 238 us (lz + 0.73) per step over lz = 2 .. 64 where
// every CTA has an SM.  The shorter last chunks fill the SMs that the full
// ones leave free.
inline double fp64_stage_cost(long tiles, int nz, int lz, int sms) {
    if (lz < 1) lz = 1;
    if (sms < 1) sms = 1;
    const double a = lz + 0.73, b = nz % lz + 0.73;  // a full chunk, the last one
    const long full = tiles * (nz / lz), rest = nz % lz ? tiles : 0;
    const long m = full / sms, x = full % sms;  // every SM has m full chunks, x of them one more
    const double cost = (double)(x ? m + 1 : m) * a;
    const long room = x ? (sms - x) * (long)(a / b) : 0;
    return rest <= room ? cost : cost + (double)((rest - room + sms - 1) / sms) * b;
}

// Cost model of one stage launch in the pair form, in plane times of a CTA
// that shares its SM with two others (2.5 us on GB300).  Three CTAs fit on an
// SM; a plane takes 0.57 with one there, 0.77 with two.  A chunk costs its
// planes plus 1.6 for its two lighter warm-up planes and its start, a launch
// 0.64.  A launch of one wave runs at the pace of its fullest SM; beyond one
// wave CTAs are handed out as they finish, so the time lies between the busiest
// SM's rounds and the even share (weighted 0.8 and 0.2).  Against the measured
// step times of cubes from 32^3 to 384^3 over 20 chunk lengths the cheapest
// pick is the fastest or within 3.6 % of it (176^3; 1 % at the others); the
// column kernel's chunk is up to 1.7x off on small ones (us per step, that
// chunk and the pick: 32^3 29.9 17.5, 48^3 30.6 23.2, 96^3 84.1 76.6, 160^3
// 328 304).
inline double pair_stage_cost(uint32_t nx, uint32_t ny, uint32_t nz, int lz, int sms) {
    if (lz < 1) lz = 1;
    if (sms < 1) sms = 1;
    const long tiles = (long)((nx + 15) / 16) * (long)((ny + 15) / 16);
    const long chunks = ((long)nz + lz - 1) / lz;
    const long lz_eff = ((long)nz + chunks - 1) / chunks;
    const long ctas = tiles * chunks;
    const long m = (ctas + sms - 1) / sms;
    const long full = (m - 1) / 3, last = m - 3 * full;
    const double rounds = (double)full + (last == 1 ? 0.57 : (last == 2 ? 0.77 : 1.0));
    const double share = (double)ctas / (3.0 * sms);
    const double waves = share <= 1.0 ? rounds : 0.8 * rounds + 0.2 * share;
    return waves * ((double)lz_eff + 1.6) + 0.64;
}

}  // namespace bubble
