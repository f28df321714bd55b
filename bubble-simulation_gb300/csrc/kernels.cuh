// CUDA kernels of the lattice time step.
//
//   init_kernel          shaders/init.wgsl:18-26
//   nucleate_kernel      shaders/nucleate.wgsl:59-85
//   prim_kernel          shaders/primitives.wgsl:16-23   (reference-structured path)
//   stage_ref_kernel     shaders/step.wgsl:92-174         (reference-structured path)
//   diag_kernel          shaders/reduce.wgsl:49-140, single pass, FP64 sums
//
// This header is included by translation units that differ only in their
// arithmetic flags (see physics.cuh); every template here is instantiated
// there.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "params.h"
#include "physics.cuh"

namespace bubble {
namespace dev {

// Start of a kernel launched as a programmatic dependent: waits until the
// launches before it have completed and their stores are visible.  Does
// nothing in a plain launch.
BUBBLE_DEV void await_previous_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// wrap1 (shaders/common.wgsl:80-89): reach <= 2 with n >= 8, one add suffices.
BUBBLE_DEV int wrap1(int i, int n) {
    int r = i;
    if (r < 0) r += n;
    if (r >= n) r -= n;
    return r;
}

template <typename R>
BUBBLE_DEV size_t cell_index(int x, int y, int z, const LatticeParams<R> &P) {
    return ((size_t)z * (size_t)P.ny + (size_t)y) * (size_t)P.nx + (size_t)x;
}

// ---------------------------------------------------------------------------
//  init (shaders/init.wgsl:18-26): phi = pi = 0, E = e_ref, Z = 0
// ---------------------------------------------------------------------------
template <typename R>
__global__ void init_kernel(V2<R> *__restrict__ field, V4<R> *__restrict__ fluid, uint64_t n,
                            R e_ref) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        field[i] = V2<R>{R(0), R(0)};
        fluid[i] = V4<R>{e_ref, R(0), R(0), R(0)};
    }
}

// ---------------------------------------------------------------------------
//  nucleate (shaders/nucleate.wgsl:59-85)
// ---------------------------------------------------------------------------
// phi <- max(phi, phi_b/2 (1 - tanh((r - r0 dx) / l_w))) over the batch, r the
// minimum-image distance from the integer cell position.  As in the
// reference the max reaches every cell: a bubble farther than the tanh
// cut-off contributes exactly 0 (det_tanh_r rounds to 1 there), so those
// terms are max(phi, 0) without evaluating tanh.
// Bubbles travel as a by-value kernel parameter (constant bank, broadcast
// to the warp), so a nucleation launch needs no staging copy; larger batches
// are split over several launches, which gives the same result because max()
// is exact and order-independent.
constexpr int kNucleateBatch = 128;
struct BubbleBatch {
    int32_t count;
    int32_t _pad[3];
    V4<float> b[kNucleateBatch];
};

// The launch covers the lattice in bricks of 32 x 8 x 8 cells, one CTA
// each.  The CTA first keeps the bubbles that can reach its brick: a lower
// bound of every cell's distance (per axis the circular distance of the
// brick's centre minus its half extent -- the periodic distance is
// 1-Lipschitz) whose tanh argument exceeds the cut-off by a margin rules a
// bubble out, its profile being exactly 0 in the whole brick.  The bound is
// evaluated in FP32 and shortened by more than its rounding: 4e-3 cells for
// axes of 2048 cells and 2e-6 of the centre's coordinates and the radius, which
// are the caller's and may lie far outside (in FP64, at two operations per clock
// and SM, the bounds alone took half of a launch of 128 bubbles).  A bound whose
// square leaves the FP32 range rules nothing out.  Every cell then takes max(phi,
// 0), the far field of all the batch's bubbles, and the maximum over the kept
// bubbles alone, in any order: the result equals the reference's loop over the
// whole batch bit for bit.  A thread's eight cells are loaded together, and a
// cell whose value does not change is not written back, so a brick out of
// reach is one read of the field.  512^3, one late bubble: 0.82 -> 0.21 ms;
// 128 bubbles: 1.53 -> 0.62 ms.
constexpr int kNucBx = 32, kNucBy = 8, kNucBz = 8;

template <typename R>
__global__ void __launch_bounds__(256) nucleate_kernel(V2<R> *__restrict__ field,
                                                        const __grid_constant__ BubbleBatch batch,
                                                        LatticeParams<R> P) {
    await_previous_launch();
    __shared__ int kept[kNucleateBatch];
    __shared__ int n_kept;
    const int bx = blockIdx.x * kNucBx, by = blockIdx.y * kNucBy, bz = blockIdx.z * kNucBz;
    const int ex = min(kNucBx, P.nx - bx), ey = min(kNucBy, P.ny - by), ez = min(kNucBz, P.nz - bz);
    if (threadIdx.x == 0) n_kept = 0;
    __syncthreads();
    const R cut = TanhCut<R>::value;
    for (int b = threadIdx.x; b < batch.count; b += blockDim.x) {
        const V4<float> bub = batch.b[b];
        const float c[3] = {bub.x, bub.y, bub.z};
        const int b0[3] = {bx, by, bz}, e[3] = {ex, ey, ez}, n[3] = {P.nx, P.ny, P.nz};
        float lb2 = 0.0f;
        for (int a = 0; a < 3; ++a) {
            const float half = 0.5f * (float)(e[a] - 1);
            float d = (float)b0[a] + half - c[a];
            if (d > 0.5f * n[a]) d -= n[a];
            if (d < -0.5f * n[a]) d += n[a];
            const float g = fmaxf(fabsf(d) - half, 0.0f);
            lb2 += g * g;
        }
        const float slack = 4e-3f + 2e-6f * (fabsf(c[0]) + fabsf(c[1]) + fabsf(c[2]) + fabsf(bub.w));
        const float arg_lb = (sqrtf(lb2) - bub.w - slack) * (float)P.dx / (float)P.wall_width;
        if (!(arg_lb > (float)cut + 0.25f && lb2 < 1e38f)) kept[atomicAdd(&n_kept, 1)] = b;
    }
    __syncthreads();
    const int nk = n_kept;
    const int tx = threadIdx.x % kNucBx, ty = threadIdx.x / kNucBx;
    if (tx >= ex || ty >= ey) return;
    const size_t i0 = cell_index(bx + tx, by + ty, bz, P), plane = (size_t)P.nx * P.ny;
    R phi_in[kNucBz];
#pragma unroll
    for (int zz = 0; zz < kNucBz; ++zz) phi_in[zz] = zz < ez ? field[i0 + zz * plane].x : R(0);
    const R nxr = R(P.nx), nyr = R(P.ny), nzr = R(P.nz);
    const R px = R(bx + tx), py = R(by + ty);
#pragma unroll
    for (int zz = 0; zz < kNucBz; ++zz) {
        if (zz >= ez) break;
        const R phi0 = phi_in[zz];
        R phi = vmax(phi0, R(0));
        const R pz = R(bz + zz);
        for (int q = 0; q < nk; ++q) {
            const V4<float> bub = batch.b[kept[q]];
            const R dx = min_image(px - R(bub.x), nxr);
            const R dy = min_image(py - R(bub.y), nyr);
            const R dz = min_image(pz - R(bub.z), nzr);
            const R r = sqrt(dx * dx + dy * dy + dz * dz) * P.dx;
            const R arg = (r - R(bub.w) * P.dx) / P.wall_width;
            R profile = R(0);
            if (!(arg > cut)) profile = R(0.5) * P.phi_b * (R(1.0) - det_tanh_r<R>(arg));
            phi = vmax(phi, profile);
        }
        bool same;
        if constexpr (sizeof(R) == 4) same = __float_as_uint((float)phi) == __float_as_uint((float)phi0);
        else same = __double_as_longlong((double)phi) == __double_as_longlong((double)phi0);
        if (!same) field[i0 + zz * plane].x = phi;
    }
}

// ---------------------------------------------------------------------------
//  Reference-structured path: primitives pass + stage pass
// ---------------------------------------------------------------------------
template <typename R>
__global__ void prim_kernel(const V4<R> *__restrict__ fluid, V4<R> *__restrict__ prim, uint64_t n,
                            LatticeParams<R> P) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        prim[i] = prim_from_cons<R, false>(fluid[i], P);
}

// One thread per cell, two HLL fluxes per axis, every operand read from
// global memory: the reference's own kernel structure (step.wgsl:92-174).
template <typename R>
__global__ void stage_ref_kernel(StageArgs<R> A, const V4<R> *__restrict__ prim,
                                 LatticeParams<R> P) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    const int z = blockIdx.z;
    if (x >= P.nx) return;
    const R zmax2 = P.z_max * P.z_max;
    const size_t i0 = cell_index(x, y, z, P);
    const V2<R> f0 = A.field_in[i0];
    const R phi0 = f0.x, pi0 = f0.y;
    const V4<R> q0 = sanitise(prim[i0], P.p_floor, zmax2);
    R lap_sum = R(0);
    R grad[3] = {R(0), R(0), R(0)};
    V4<R> fd{R(0), R(0), R(0), R(0)};
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
        const int ex = axis == 0, ey = axis == 1, ez = axis == 2;
        const size_t im1 = cell_index(wrap1(x - ex, P.nx), wrap1(y - ey, P.ny), wrap1(z - ez, P.nz), P);
        const size_t ip1 = cell_index(wrap1(x + ex, P.nx), wrap1(y + ey, P.ny), wrap1(z + ez, P.nz), P);
        const size_t im2 =
            cell_index(wrap1(x - 2 * ex, P.nx), wrap1(y - 2 * ey, P.ny), wrap1(z - 2 * ez, P.nz), P);
        const size_t ip2 =
            cell_index(wrap1(x + 2 * ex, P.nx), wrap1(y + 2 * ey, P.ny), wrap1(z + 2 * ez, P.nz), P);
        const R phi_m = A.field_in[im1].x;
        const R phi_p = A.field_in[ip1].x;
        lap_sum = lap_sum + (phi_m + phi_p - R(2.0) * phi0);
        grad[axis] = R(0.5) * (phi_p - phi_m) * P.inv_dx;
        const V4<R> qm2 = sanitise(prim[im2], P.p_floor, zmax2);
        const V4<R> qm1 = sanitise(prim[im1], P.p_floor, zmax2);
        const V4<R> qp1 = sanitise(prim[ip1], P.p_floor, zmax2);
        const V4<R> qp2 = sanitise(prim[ip2], P.p_floor, zmax2);
        const V4<R> s_m1 = limit_slope4(v4_sub(qm1, qm2), v4_sub(q0, qm1));
        const V4<R> s_0 = limit_slope4(v4_sub(q0, qm1), v4_sub(qp1, q0));
        const V4<R> s_p1 = limit_slope4(v4_sub(qp1, q0), v4_sub(qp2, qp1));
        const V4<R> lm = sanitise(half_step(qm1, s_m1, R(1)), P.p_floor, zmax2);
        const V4<R> rm = sanitise(half_step(q0, s_0, R(-1)), P.p_floor, zmax2);
        const V4<R> lp = sanitise(half_step(q0, s_0, R(1)), P.p_floor, zmax2);
        const V4<R> rp = sanitise(half_step(qp1, s_p1, R(-1)), P.p_floor, zmax2);
        V4<R> fm, fp;
        if (axis == 0) {
            fm = hll_flux<0, R, false, kPlain, false>(lm, rm, zmax2, P);
            fp = hll_flux<0, R, false, kPlain, false>(lp, rp, zmax2, P);
        } else if (axis == 1) {
            fm = hll_flux<1, R, false, kPlain, false>(lm, rm, zmax2, P);
            fp = hll_flux<1, R, false, kPlain, false>(lp, rp, zmax2, P);
        } else {
            fm = hll_flux<2, R, false, kPlain, false>(lm, rm, zmax2, P);
            fp = hll_flux<2, R, false, kPlain, false>(lp, rp, zmax2, P);
        }
        fd.x = fd.x + (fp.x - fm.x) * P.inv_dx;
        fd.y = fd.y + (fp.y - fm.y) * P.inv_dx;
        fd.z = fd.z + (fp.z - fm.z) * P.inv_dx;
        fd.w = fd.w + (fp.w - fm.w) * P.inv_dx;
    }
    const R laplacian = lap_sum * P.inv_dx * P.inv_dx;
    const R vv = q0.x * q0.x + q0.y * q0.y + q0.z * q0.z;
    const R gam = R(1.0) / sqrt(vmax(R(1.0) - vv, R(1e-12)));
    const R dphi_proper = gam * (pi0 + (q0.x * grad[0] + q0.y * grad[1] + q0.z * grad[2]));
    const R drag = P.eta * dphi_proper;
    const R d_phi = pi0;
    const R d_pi = laplacian - dpotential(phi0, P) - drag;
    const R dE = -fd.x + drag * pi0;
    const R dZx = -fd.y - drag * grad[0];
    const R dZy = -fd.z - drag * grad[1];
    const R dZz = -fd.w - drag * grad[2];
    const V4<R> u_in = A.fluid_in[i0];
    const V2<R> fu{f0.x + A.dt * d_phi, f0.y + A.dt * d_pi};
    const V4<R> uu{u_in.x + A.dt * dE, u_in.y + A.dt * dZx, u_in.z + A.dt * dZy,
                   u_in.w + A.dt * dZz};
    if (A.stage == 0) {
        A.field_out[i0] = V2<R>{A.a1 * fu.x, A.a1 * fu.y};
        A.fluid_out[i0] = V4<R>{A.a1 * uu.x, A.a1 * uu.y, A.a1 * uu.z, A.a1 * uu.w};
    } else {
        const V2<R> fn = A.field_n[i0];
        const V4<R> un = A.fluid_n[i0];
        A.field_out[i0] = V2<R>{A.a0 * fn.x + A.a1 * fu.x, A.a0 * fn.y + A.a1 * fu.y};
        A.fluid_out[i0] = V4<R>{A.a0 * un.x + A.a1 * uu.x, A.a0 * un.y + A.a1 * uu.y,
                                A.a0 * un.z + A.a1 * uu.z, A.a0 * un.w + A.a1 * uu.w};
    }
}

// ---------------------------------------------------------------------------
//  Diagnostics (shaders/reduce.wgsl:49-140), one pass, FP64 sums
// ---------------------------------------------------------------------------
// Per-cell terms in the state precision exactly as cell_contribution; sums in
// FP64.  Every block writes its partial to `partials`; the last block to
// finish (ticket counter) folds them in a fixed order, writes `out` and
// re-arms the counter, so the result does not depend on block timing.  `out`
// and `status_out` may be pinned host memory: the report and the bounded
// waits' status word then arrive with the launch, without a copy (64^3 37 ->
// 26 us a report).
//
// Work item: 256 cells of a plane, one per thread, marched through a chunk of
// z planes with phi of the planes around z carried in registers, so a cell's
// position is decoded once per item and the field and fluid are read once.
//
// What bounded it (3.24 ms a report at 512^3, 0.47 ms of traffic): IEEE
// divisions with zero or tiny numerators, which leave the fast path
// (div_scaled: 2.27 -> 1.29 ms at four blocks per SM), residency (2.07 -> 1.29
// ms) and the FP64 pipe, which adds two doubles per clock and SM (0.4 ms).  An
// FP32 state's terms are summed over a chunk as unevaluated pairs hi + lo
// (Knuth's TwoSum; lo collects the exact rounding errors of hi) and the pair
// is added in FP64 once per chunk; cells of the broken phase are counted.  lo
// is a sum of at most 32 terms below 2^-24 hi, so a chunk's pair is within
// 2^-44 of exact, unbiased, and the total over many chunks well below that
// (the fluid energies of 64^3 to 256^3 states sum to the correctly rounded
// double).  A chunk whose sums leave the FP32 range (terms above 1e37,
// infinities, NaN) is marched again with each term added in FP64 (in code of its
// own: 512^3 1.34 -> 1.37 ms; a flag in the loop: 1.48).  The largest speed is taken from the largest |v|^2 (sqrt is
// monotone).  Now 1.27 ms at 512^3, bound by instruction issue; 256^3 0.59 ->
// 0.21 ms, 128^3 96 -> 60 us.
constexpr int kDiagThreads = 256;
constexpr int kDiagMaxBlocks = 1024;

struct DiagPartial {
    double s[4];
    float vmax;
    uint32_t nonfinite;
    uint32_t _pad[2];
};

template <typename R>
BUBBLE_DEV double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

constexpr int kDiagBlocksPerSm = 4;  // at 512^3: 2.07 ms with 3, 1.29 with 4, 1.40 with 5, 1.66 with 8

// Planes of a chunk.  Bag forms in FP32: about two items per SM on small lattices
// (one round of blocks: 64^3 58 us a report at one plane, 39 at four), at most
// 32 planes.  The Newton steps of the gamma law and the thermal potential and
// the FP64 pipe make a plane several times as long, so there the even share of
// the SMs decides and long items end unevenly (us a report, the bag forms' rule
// and this one: gamma law 112^3 188 and 88, 128^3 306 and 163, 160^3 517 and 345,
// 256^3 1271 and 1157; thermal potential 128^3 354 and 193; FP64 128^3 628 and
// 517).  One plane up to 12288 plane groups: two planes take 284 us at 144^3
// where one takes 244, and 345 at 160^3 where one takes 339 (on a lattice full
// of walls 143 and 164).
template <typename R, int MIXED>
inline int diag_planes(uint64_t nx, uint64_t ny, uint64_t nz) {
    const uint64_t groups = (nx * ny + kDiagThreads - 1) / kDiagThreads * nz;  // 256 cells of a plane each
    const int lz = groups > 32 * 300 ? 32 : (int)((groups + 299) / 300);
    if (sizeof(R) == 8) return groups > 1200 ? 3 : lz;
    if (MIXED == kGamma || MIXED == kThermal) return groups > 12288 ? 2 : (groups > 4096 ? 1 : (lz < 4 ? lz : 4));
    return lz;
}

// A sum of FP32 terms as hi + lo, or of doubles.
template <typename R>
struct TermSum {
    R hi = R(0), lo = R(0);
    BUBBLE_DEV void add(R x) {
        if constexpr (sizeof(R) == 4) {
            const R s = hi + x;
            const R b = s - hi;
            lo = lo + ((hi - (s - b)) + (x - b));
            hi = s;
        } else {
            hi += x;
        }
    }
};

// a / b for a normal b > 0, kept on IEEE division's fast path: a zero or tiny a,
// common in the fluid at rest ahead of the walls, goes to a subroutine there and
// splits its warp.  The scaling is exact; a quotient below 2^-126 is rounded
// twice, and every such quotient is squared or added to the energy density,
// where it is far below rounding.
BUBBLE_DEV float div_scaled(float a, float b) {
    const bool small = fabsf(a) < 1.0f;
    const float n = a == 0.0f ? 1.0f : a * (small ? 0x1p48f : 1.0f);
    const float q = n / b * (small ? 0x1p-48f : 1.0f);
    return a == 0.0f ? a : q;
}

// recover<R, false, MIXED>(u, P, phi) with those divisions.
template <typename R, int MIXED>
BUBBLE_DEV V4<R> diag_recover(const V4<R> &u, const LatticeParams<R> &P, R phi) {
    if constexpr (sizeof(R) == 4 && (MIXED == kPlain || MIXED == kMixed || MIXED == kPert)) {
        const float de = vmax(u.x, P.e_floor);
        const float e_lab = MIXED == kPert ? P.e_bg + de : de;
        float zx = u.y, zy = u.z, zz = u.w;
        const float zcap = P.z_max * e_lab;
        V4<float> q;
        if constexpr (MIXED == kPert) {
            const float z2 = capped_z2(zx, zy, zz, zcap);
            const float sq = sqrt(vmax(4.0f * e_lab * e_lab - 3.0f * z2, 0.0f));
            const float dp = vmax(div_scaled(de, 3.0f) - div_scaled(z2, sq + 2.0f * e_lab), P.p_floor);
            const float d = vmax(e_lab + P.p_bg + dp, 1e-30f);
            q = V4<float>{div_scaled(zx, d), div_scaled(zy, d), div_scaled(zz, d), dp};
        } else {
            const PrimParts<float> r = prim_parts(e_lab, zx, zy, zz, zcap, P);
            q = V4<float>{div_scaled(r.zx, r.s), div_scaled(r.zy, r.s), div_scaled(r.zz, r.s), r.p};
        }
        if constexpr (MIXED != kPlain) {
            if (q.x * q.x + q.y * q.y + q.z * q.z > 8.0f / 9.0f) return recover<R, false, MIXED>(u, P, phi);
        }
        return q;
    } else {
        return recover<R, false, MIXED>(u, P, phi);
    }
}
// potential(phi, P) likewise
template <typename R>
BUBBLE_DEV R diag_potential(R phi, const LatticeParams<R> &P) {
    if constexpr (sizeof(R) == 4) {
        const R p2 = phi * phi;
        return 0.5f * P.m2 * p2 - div_scaled(P.delta * p2 * phi, 3.0f) + 0.25f * P.lambda * p2 * p2;
    } else {
        return potential(phi, P);
    }
}

template <typename R, int MIXED>
__global__ void __launch_bounds__(kDiagThreads, kDiagBlocksPerSm)
    diag_kernel(const V2<R> *__restrict__ field, const V4<R> *__restrict__ fluid,
                LatticeParams<R> P, DiagPartial *__restrict__ partials,
                unsigned int *__restrict__ ticket, DiagResult *__restrict__ out, const int *__restrict__ status,
                int *__restrict__ status_out, int lz) {
    await_previous_launch();
    const uint64_t n = (uint64_t)P.nx * P.ny * P.nz;
    const uint32_t plane = (uint32_t)P.nx * (uint32_t)P.ny;
    const uint32_t groups = (plane + kDiagThreads - 1) / kDiagThreads;
    const uint32_t items = groups * (uint32_t)((P.nz + lz - 1) / lz);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    R v2max = R(0);
    uint32_t bad = 0;
    for (uint32_t it = blockIdx.x; it < items; it += gridDim.x) {
        const uint32_t chunk = it / groups;
        const uint32_t c = (it - chunk * groups) * kDiagThreads + threadIdx.x;
        if (c >= plane) continue;
        const int y = (int)(c / (uint32_t)P.nx), x = (int)(c - (uint32_t)y * (uint32_t)P.nx);
        // in-plane neighbours, periodic
        const uint32_t cxp = x + 1 < P.nx ? c + 1 : c + 1 - P.nx, cxm = x > 0 ? c - 1 : c - 1 + P.nx;
        const uint32_t cyp = y + 1 < P.ny ? c + P.nx : c + P.nx - plane, cym = y > 0 ? c - P.nx : c - P.nx + plane;
        const int z0 = (int)chunk * lz, z1 = min(z0 + lz, P.nz);
        TermSum<R> s_total, s_kinetic, s_e;
        // The chunk's terms into the pairs, or (WIDE) each into the FP64 sums;
        // returns its cells in the broken phase.
        auto march = [&](auto wide) {
            constexpr bool WIDE = decltype(wide)::value;
            // cell indices fit 32 bits
            R phi_m = field[(uint32_t)wrap1(z0 - 1, P.nz) * plane + c].x;
            V2<R> f = field[(uint32_t)z0 * plane + c];
            uint32_t broken = 0;
#pragma unroll 1
            for (int z = z0; z < z1; ++z) {
                const uint32_t pl = (uint32_t)z * plane;
                const V2<R> f_p = field[(uint32_t)wrap1(z + 1, P.nz) * plane + c];
                const V4<R> u = fluid[pl + c];
                const R phi = f.x, pi = f.y;
                R grad2 = R(0);
                {
                    const R d = R(0.5) * (field[pl + cxp].x - field[pl + cxm].x) * P.inv_dx;
                    grad2 = grad2 + d * d;
                }
                {
                    const R d = R(0.5) * (field[pl + cyp].x - field[pl + cym].x) * P.inv_dx;
                    grad2 = grad2 + d * d;
                }
                {
                    const R d = R(0.5) * (f_p.x - phi_m) * P.inv_dx;
                    grad2 = grad2 + d * d;
                }
                // In the perturbation form e_lab is max(E, e_floor) - e_bg: the sums of
                // e_total and e_lab then miss N e_bg, which the host adds in FP64.
                const R e_lab = vmax(u.x, P.e_floor);
                const V4<R> q = diag_recover<R, MIXED>(u, P, phi);
                const R v2 = q.x * q.x + q.y * q.y + q.z * q.z;
                // the thermal form's field holds V(phi, 0); the rest of V(phi, T) is in E
                R pot;
                if constexpr (MIXED == kThermal) pot = thermal_potential0(phi, P);
                else pot = diag_potential(phi, P);
                const R e_total = R(0.5) * pi * pi + R(0.5) * grad2 + pot + e_lab;
                R kinetic;
                if constexpr (MIXED == kPert) kinetic = ((e_lab + q.w) + (P.e_bg + P.p_bg)) * v2;
                else kinetic = (e_lab + q.w) * v2;
                if constexpr (!WIDE) {
                    s_total.add(e_total);
                    s_kinetic.add(kinetic);
                    s_e.add(e_lab);
                } else {
                    acc[0] += (double)e_total;
                    acc[2] += (double)kinetic;
                    acc[3] += (double)e_lab;
                }
                broken += phi > R(0.5) * P.phi_b ? 1u : 0u;
                v2max = vmax(v2max, v2);
                // max(E, e_floor) hides a NaN in E, so the raw state is checked too.
                if (!isfinite(e_total) || !isfinite(v2) || !isfinite(f.x + f.y + u.x + u.y + u.z + u.w)) bad = 1;
                phi_m = phi;
                f = f_p;
            }
            return broken;
        };
        acc[1] += (double)march(std::false_type{});
        if (sizeof(R) == 4 && !isfinite(s_total.hi + s_kinetic.hi + s_e.hi)) {
            march(std::true_type{});
        } else {
            acc[0] += (double)s_total.hi + (double)s_total.lo;
            acc[2] += (double)s_kinetic.hi + (double)s_kinetic.lo;
            acc[3] += (double)s_e.hi + (double)s_e.lo;
        }
    }
    float vmaxv = (float)sqrt(v2max);
    if (!isfinite(vmaxv)) bad = 1;
    __shared__ double sh[kDiagThreads / 32][4];
    __shared__ float shm[kDiagThreads / 32];
    __shared__ uint32_t shb[kDiagThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = warp_sum<R>(acc[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        vmaxv = fmaxf(vmaxv, __shfl_xor_sync(0xffffffffu, vmaxv, o));
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    if (lane == 0) {
        for (int k = 0; k < 4; ++k) sh[w][k] = acc[k];
        shm[w] = vmaxv;
        shb[w] = bad;
    }
    __syncthreads();
    __shared__ bool last;
    if (threadIdx.x == 0) {
        DiagPartial pt;
        for (int k = 0; k < 4; ++k) {
            double s = 0.0;
            for (int q = 0; q < kDiagThreads / 32; ++q) s += sh[q][k];
            pt.s[k] = s;
        }
        float m = 0.0f;
        uint32_t b = 0;
        for (int q = 0; q < kDiagThreads / 32; ++q) {
            m = fmaxf(m, shm[q]);
            b |= shb[q];
        }
        pt.vmax = m;
        pt.nonfinite = b;
        pt._pad[0] = pt._pad[1] = 0;
        partials[blockIdx.x] = pt;
        __threadfence();
        const unsigned int prev = atomicAdd(ticket, 1u);
        last = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // Fold the partials: thread k sums partials k, k+256, ... in order, then
    // a fixed tree over the 256 threads.
    __shared__ double fold[kDiagThreads][4];
    __shared__ float foldm[kDiagThreads];
    __shared__ uint32_t foldb[kDiagThreads];
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    float m = 0.0f;
    uint32_t b = 0;
    for (unsigned q = threadIdx.x; q < gridDim.x; q += blockDim.x) {
        const volatile DiagPartial *pp = partials + q;
        for (int k = 0; k < 4; ++k) s[k] += pp->s[k];
        m = fmaxf(m, pp->vmax);
        b |= pp->nonfinite;
    }
    for (int k = 0; k < 4; ++k) fold[threadIdx.x][k] = s[k];
    foldm[threadIdx.x] = m;
    foldb[threadIdx.x] = b;
    __syncthreads();
    for (int h = kDiagThreads / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            for (int k = 0; k < 4; ++k) fold[threadIdx.x][k] += fold[threadIdx.x + h][k];
            foldm[threadIdx.x] = fmaxf(foldm[threadIdx.x], foldm[threadIdx.x + h]);
            foldb[threadIdx.x] |= foldb[threadIdx.x + h];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < 4; ++k) out->sums[k] = fold[0][k];
        out->max_v_bits = __float_as_uint(foldm[0]);
        out->nonfinite = foldb[0];
        out->cells = n;
        if (status_out) *status_out = *status;
        *ticket = 0u;  // re-arm for the next launch on this scratch
    }
}

// One block per item, at most the blocks that `sms` SMs hold.
inline int diag_blocks(uint64_t nx, uint64_t ny, uint64_t nz, uint64_t lz, int sms) {
    const uint64_t items = (nx * ny + kDiagThreads - 1) / kDiagThreads * ((nz + lz - 1) / lz);
    uint64_t most = (uint64_t)kDiagBlocksPerSm * (uint64_t)(sms > 0 ? sms : 1);
    if (most > (uint64_t)kDiagMaxBlocks) most = kDiagMaxBlocks;
    return (int)(items < most ? items : most);
}

}  // namespace dev
}  // namespace bubble
