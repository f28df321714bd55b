// Fused SSP-RK3 stage kernel, pair form: the fast arithmetic (FP32, every
// form and equation of state) on 16 x 16 tiles.
//
// The scheme of stage_column.cuh (z-marching column tile, three phases and
// two barriers per plane, TMA-staged raw planes) with two cells per thread:
// column thread (ci, cj), cj < 8, owns the cells (ci, cj) and (ci, cj + 8) of
// its tile as the halves of float2 values (physics_pair.cuh).  A plane of
// primitives, fluxes or face states in shared memory holds "pair rows": pair
// row j is the rows j and j + 8, so a neighbour in x or y is one pair away
// for both halves.  Rows 7 and 8 are each wanted in two pair rows (7 and -1,
// 8 and 0) and are stored twice.
//
// Four column warps and one halo warp make a CTA.  The halo warp recovers the
// tile's halo ring and computes the face states and fluxes on the tile's far
// edges: two ring pairs, one face-state pair and half a flux pair per plane
// and thread, about what a column thread does.
//
// What bounds it.  The scalar column form issued 26.6 warp instructions per
// cell and stage (256^3, MIXED) and was bound by that; the pair form issues
// 16.4 (15.6 in the first stage).  Packed FP32 takes the FMA pipe as long as two scalar instructions
// (0.36 fma.f32x2 and 0.49 add.f32x2 or mul.f32x2 per clock and scheduler,
// measured, against 0.61 fma and 0.93 add), so it saves issue slots, not
// arithmetic time: FMA pipe 50 %, shared-memory data path 63 %, issue 59 % at
// 14 warps per SM, the rest dependency latency and barriers.  Registers set
// the residency: 15 warps over four schedulers leave 128 per thread.  Measured
// and not kept: 16 warps in four CTAs without a halo warp (equal on large
// lattices, slower below 160^3), the axes on separate warps at 72 registers
// (barrier-bound), U_in and U^n loaded at the combine (8 % slower), the march
// unrolled by 2 or 3 (20 to 30 % slower), the plane barriers split into
// mbarrier arrivals and waits around independent work (1 to 4 % slower), the
// first stage in its own instantiation (1 % faster from 128^3, 1 % slower at
// 64^3 and below, where two kernels alternate).  Step time, column form to
// pair form (GB300): 512^3 MIXED 10.85 -> 8.26 ms, 256^3 perturbation 1.54 ->
// 1.16 ms, 128^3 0.212 -> 0.170 ms, 64^3 49.3 -> 43.1 us (0.160 ms and 36.5 us
// with dependent launches and the form's own z chunk); the gamma law at 128^3,
// with its recovery in closed form, 0.33 -> 0.18 ms, the thermal potential at
// 96^3, with its short iterations, 0.374 -> 0.177 ms (0.240 at two CTAs per SM,
// where it has no spills).
//
// Every tile is processed in full: a tile that reaches past the lattice
// stages the wrapped cells beyond the edge, so the faces and neighbours of
// the last row and column come out of the same code, and only the combine is
// masked.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "kernels.cuh"
#include "physics_pair.cuh"
#include "staging.cuh"
#include "tma.h"

namespace bubble {
namespace dev {

struct PairLayout {
    static constexpr int TX = 16, TY = 16;
    static constexpr int PW = TX + 4, PC = PW * (TY + 4);  // raw plane, cells
    // primitive and phi planes, pairs (pair rows -2 .. 9); the odd pitch keeps
    // the halo warp's column accesses free of bank conflicts
    static constexpr int PQ = PW + 1, PP = PQ * (TY / 2 + 4);
    static constexpr int NC = TX * TY / 2, NT = NC + 32;
    static constexpr int MIN_BLOCKS = 3;
    // x faces of a plane [j][i], i = 0 .. 16, and y faces [j][i], j = 0 .. 8
    static constexpr int FXW = TX + 1, FX = (TY / 2) * FXW, FY = (TY / 2 + 1) * TX;
    // shared memory map (bytes); a pair array is two float4 arrays, of the (x,
    // y) and of the (z, w) components
    static constexpr size_t o_rawu = 0;
    static constexpr size_t o_rawf = align128(o_rawu + 2 * PC * sizeof(float4));
    static constexpr size_t o_prim = align128(o_rawf + 2 * PC * sizeof(float2));  // primitives of plane z
    static constexpr size_t o_phi = o_prim + 2 * PP * sizeof(float4);             // phi, 4 slots
    static constexpr size_t o_hx = align128(o_phi + 4 * PP * sizeof(float2));     // upper states at x faces
    static constexpr size_t o_hy = o_hx + 2 * FX * sizeof(float4);
    static constexpr size_t o_fx = o_hy + 2 * FY * sizeof(float4);  // fluxes
    static constexpr size_t o_fy = o_fx + 2 * FX * sizeof(float4);
    static constexpr size_t o_lx = o_fy + 2 * FY * sizeof(float4);        // lower x states of column 16
    static constexpr size_t o_ly = o_lx + 2 * (TY / 2) * sizeof(float4);  // [i] lower y state of row 16 (one cell)
    static constexpr size_t o_bar = o_ly + TX * sizeof(float4);
    static constexpr size_t o_dead = o_bar + 2 * sizeof(uint64_t);
    static constexpr size_t bytes = o_dead + 4 * sizeof(int);
    static constexpr uint32_t plane_tx_bytes = PC * (sizeof(float4) + sizeof(float2));
};

BUBBLE_DEV void plane_barrier() { asm volatile("bar.sync 0;" ::: "memory"); }
BUBBLE_DEV void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// Planes that U^n is fetched ahead: it comes from DRAM (U_in is in L2, its
// planes were just staged); 512^3 4 % faster, 1 and 4 planes measured the same.
constexpr int kAhead = 2;

// A pair stored as two float4 arrays N apart, at place c.
template <int N>
BUBBLE_DEV P4 get_pair(const float4 *a, int c) {
    return pair_of(a[c], a[c + N]);
}
template <int N>
BUBBLE_DEV void put_pair(float4 *a, int c, const P4 &q) {
    a[c] = pair_a(q);
    a[c + N] = pair_b(q);
}
// Half FROM of a pair alone, into half TO of place c.
template <int N, int FROM, int TO>
BUBBLE_DEV void put_half(float4 *a, int c, const P4 &q) {
    float *u = reinterpret_cast<float *>(a + c) + TO, *v = reinterpret_cast<float *>(a + c + N) + TO;
    u[0] = FROM ? q.x.y : q.x.x;
    u[2] = FROM ? q.y.y : q.y.x;
    v[0] = FROM ? q.z.y : q.z.x;
    v[2] = FROM ? q.w.y : q.w.x;
}

// Stage combine of one cell of a pair: u1 = U_in + dt L, out = U^n + a1 (u1 -
// U^n), whose weights sum to 1 exactly; u1 in the first stage, whose a1 is 1.
// The last stage rounds u1 on its own: U^n + a1 (dt L + (U_in - U^n)), with
// one rounding less, drops every increment below 3/4 ulp where rounding u1
// drops those below 1/2, and left twice the error in E and Z after 100 steps of
// 128^3.  Cells of the mixed form beyond gamma = 3 (om = 1 - v^2 below 1/9),
// which magnify the rounding of E and Z, take the order with one rounding
// less in the middle stage.  Over 200 random states of speeds up to 0.999
// (errors against 64 bits after two steps, geometric mean with it over
// without) the largest errors are 0.95 in E and Z and 0.90 in pi, the root mean
// squares 0.96 and 0.93; up to 0.99, 1.01, 0.85, 0.99 and 0.91.  In every cell it
// would raise the energy's drift over 3000 steps (256^3: 6.8e-8 of it beyond
// FP64's, 8.9e-8 with every cell).  512^3 8.16 -> 8.25 ms.
template <int FORM>
BUBBLE_DEV void store_cell(const StageArgs<float> &A, uint32_t g, const V2<float> &pf, const V4<float> &pu,
                           const V2<float> &pfn, const V4<float> &pun, float d_pi, float d_e, float d_x, float d_y,
                           float d_z, float om) {
    const float dt = A.dt;
    if (A.stage == 0) {
        A.field_out[g] = V2<float>{__fmaf_rn(dt, pf.y, pf.x), __fmaf_rn(dt, d_pi, pf.y)};
        A.fluid_out[g] = V4<float>{__fmaf_rn(dt, d_e, pu.x), __fmaf_rn(dt, d_x, pu.y), __fmaf_rn(dt, d_y, pu.z),
                                   __fmaf_rn(dt, d_z, pu.w)};
    } else {
        const float a1 = A.a1;
        auto comb = [&](float d, float u, float n) { return __fmaf_rn(a1, __fsub_rn(__fmaf_rn(dt, d, u), n), n); };
        A.field_out[g] = V2<float>{comb(pf.y, pf.x, pfn.x), comb(d_pi, pf.y, pfn.y)};
        const bool mid = FORM == kMixed && A.stage == 1 && om < 1.0f / 9.0f;
        auto comb_u = [&](float d, float u, float n) {
            const float two = __fsub_rn(__fmaf_rn(dt, d, u), n), one = __fmaf_rn(dt, d, __fsub_rn(u, n));
            return __fmaf_rn(a1, mid ? one : two, n);
        };
        A.fluid_out[g] = V4<float>{comb_u(d_e, pu.x, pun.x), comb_u(d_x, pu.y, pun.y), comb_u(d_y, pu.z, pun.z),
                                   comb_u(d_z, pu.w, pun.w)};
    }
}

// One work item: the 16 x 16 tile `tile_xy`, z chunk `chunk` (planes
// [chunk*lz, min((chunk+1)*lz, nz))), one RK stage.  As column_item: returns
// false when a bounded wait expired (bit 0 of *status is set), usable
// repeatedly by one CTA.
template <int FORM>
BUBBLE_DEV bool pair_item(unsigned char *smem, const StageArgs<float> &A, const LatticeParams<float> &P, int lz,
                          const StageMaps *maps, int tma_ok, int *status, int tile_xy, int chunk) {
    using L = PairLayout;
    constexpr int PW = L::PW, PQ = L::PQ, PP = L::PP, PC = L::PC, FXW = L::FXW, FX = L::FX, FY = L::FY;
    __syncthreads();  // a previous item on this CTA is done with shared memory
    V4<float> *raw_u = reinterpret_cast<V4<float> *>(smem + L::o_rawu);
    V2<float> *raw_f = reinterpret_cast<V2<float> *>(smem + L::o_rawf);
    float4 *pr = reinterpret_cast<float4 *>(smem + L::o_prim);
    float2 *phi_s = reinterpret_cast<float2 *>(smem + L::o_phi);
    float4 *hx = reinterpret_cast<float4 *>(smem + L::o_hx);
    float4 *hy = reinterpret_cast<float4 *>(smem + L::o_hy);
    float4 *fx = reinterpret_cast<float4 *>(smem + L::o_fx);
    float4 *fy = reinterpret_cast<float4 *>(smem + L::o_fy);
    float4 *lx = reinterpret_cast<float4 *>(smem + L::o_lx);
    float4 *ly = reinterpret_cast<float4 *>(smem + L::o_ly);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + L::o_bar);
    volatile int *dead = reinterpret_cast<volatile int *>(smem + L::o_dead);  // a bounded wait of this CTA expired

    const int t = threadIdx.x;
    const int ntx = (P.nx + 15) >> 4;
    const int x0 = (tile_xy % ntx) << 4;
    const int y0 = (tile_xy / ntx) << 4;
    const int z0 = chunk * lz;
    const int z1 = min(z0 + lz, P.nz);
    const int xe = min(16, P.nx - x0);
    const int ye = min(16, P.ny - y0);
    const float zmax2 = P.z_max * P.z_max;
    // cell indices fit 32 bits: the host rejects lattices of 2^32 cells or more
    const uint32_t plane = (uint32_t)P.nx * (uint32_t)P.ny;
    const bool tma = tma_ok && x0 >= 2 && x0 + 18 <= P.nx && y0 >= 2 && y0 + 18 <= P.ny;
    const int zlast = z1 + 1;  // last plane whose primitives are needed

    // Ring slots: phi of planes z-1 .. z+2 (4 slots), raw planes z+3, z+4 (2
    // slots); p >= z0 - 2.
    auto phi_slot = [&](int p) { return phi_s + ((p - z0 + 4) & 3) * PP; };
    auto raw_slot = [&](int p) { return (p - z0) & 1; };
    // in-plane offset of the tile's cell (i, j), wrapped: the tile may reach
    // past a lattice edge by up to a tile and a halo
    auto wrapped = [&](int i, int j) {
        int x = x0 + i, y = y0 + j;
        x = x < 0 ? x + P.nx : x % P.nx;
        y = y < 0 ? y + P.ny : y % P.ny;
        return (uint32_t)y * (uint32_t)P.nx + (uint32_t)x;
    };

    // The warp index read through a shuffle is known to be warp-uniform, so
    // loop counters, slots and constants stay in the uniform registers.
    const int warp = __shfl_sync(0xffffffffu, t >> 5, 0);
    const bool col = warp < L::NC / 32;
    // Column thread: the cells (ci, cj) and (ci, cj + 8), rc and rc + 8 PW in a
    // raw plane, pair pc in a primitive plane.  Halo thread: two ring pairs;
    // pair 0 is column hi in {-2, -1, 16, 17} of the rows hj, hj + 8, pair 1
    // the rows k - 2 and 17 - k of column h & 15, k = h >> 4.
    const int h = t & 31;
    const int ci = t & 15, cj = t >> 4;
    const int hi = (h >> 3) < 2 ? (h >> 3) - 2 : 14 + (h >> 3), hj = h & 7;
    const int rc = col ? (cj + 2) * PW + ci + 2 : (hj + 2) * PW + hi + 2;
    const int pc = col ? (cj + 2) * PQ + ci + 2 : (hj + 2) * PQ + hi + 2;
    const int r1a = (h >> 4) * PW + (h & 15) + 2, r1b = (19 - (h >> 4)) * PW + (h & 15) + 2;
    const int p1a = (h >> 4) * PQ + (h & 15) + 2, p1b = (11 - (h >> 4)) * PQ + (h & 15) + 2;  // pair rows k - 2, 9 - k
    uint32_t g0, g1, g2 = 0, g3 = 0;  // in-plane offsets: own cells, or the four ring cells
    if (col) {
        g0 = wrapped(ci, cj);
        g1 = wrapped(ci, cj + 8);
    } else {
        g0 = wrapped(hi, hj);
        g1 = wrapped(hi, hj + 8);
        g2 = wrapped(h & 15, (h >> 4) - 2);
        g3 = wrapped(h & 15, 17 - (h >> 4));
    }

    if (t == 0) {
        *dead = 0;
        if (tma) {
            mbar_init(&bar[0], 1);
            mbar_init(&bar[1], 1);
            fence_mbar_init();
        }
    }
    __syncthreads();  // publishes the mbarrier initialisation

    // Stage raw plane p asynchronously into its slot.
    auto issue = [&](int p) {
        const int s = raw_slot(p);
        const int gz = wrap1(p, P.nz);
        if (tma) {
            if (t == 0) {
                fence_proxy_async();
                if (A.test_tx != 0 && p == z0) {
                    // test hook: bytes that no copy delivers, and no copy issued
                    mbar_expect_tx(&bar[s], A.test_tx);
                } else {
                    mbar_expect_tx(&bar[s], L::plane_tx_bytes);
                    tma_load_4d(raw_u + s * PC, &maps->fluid, &bar[s], 0, x0 - 2, y0 - 2, gz);
                    tma_load_3d(raw_f + s * PC, &maps->field, &bar[s], 2 * (x0 - 2), y0 - 2, gz);
                }
            }
        } else {
            const uint32_t base = (uint32_t)gz * plane;
            V4<float> *ru = raw_u + s * PC;
            V2<float> *rf = raw_f + s * PC;
            cp_async_16(ru + rc, A.fluid_in + (base + g0));
            cp_async_8(rf + rc, A.field_in + (base + g0));
            cp_async_16(ru + rc + 8 * PW, A.fluid_in + (base + g1));
            cp_async_8(rf + rc + 8 * PW, A.field_in + (base + g1));
            if (!col) {
                cp_async_16(ru + r1a, A.fluid_in + (base + g2));
                cp_async_8(rf + r1a, A.field_in + (base + g2));
                cp_async_16(ru + r1b, A.fluid_in + (base + g3));
                cp_async_8(rf + r1b, A.field_in + (base + g3));
            }
            cp_async_commit();
        }
    };
    // Wait for raw plane p (`newer`: plane p+1 was issued after it); false
    // when the bounded wait expired.
    auto wait_raw = [&](int p, bool newer) -> bool {
        if (tma) return mbar_wait_bounded(&bar[raw_slot(p)], ((p - z0) >> 1) & 1, A.wait_shift);
        if (newer) cp_async_wait_but_one();
        else cp_async_wait_all();
        return true;
    };

    issue(z0);
    issue(z0 + 1);  // zlast >= z0 + 2

    // Each role has its own march, so that neither's registers are held
    // through the other's code.  A thread whose bounded wait expires in
    // iteration z sets *dead; it is read at the top of iteration z+1, which
    // passes a barrier before any thread can set it again, so all agree.
    int stop = z1;  // iteration at whose top the march stopped
    if (col) {
        // ---- column warps ----------------------------------------------------------
        // q0, q1 = primitives of planes z, z+1; hiz = upper z state of plane z;
        // fz_m = flux of face z-1/2.  The warm-up planes z0-2, z0-1 come straight
        // from global memory.
        const float2 zero = make_float2(0.0f, 0.0f);
        P4 q0, q1, hiz{zero, zero, zero, zero}, fz_m = hiz;
        {
            const uint32_t pa = (uint32_t)wrap1(z0 - 2, P.nz) * plane, pb = (uint32_t)wrap1(z0 - 1, P.nz) * plane;
            const V4<float> a0 = A.fluid_in[pa + g0], a1 = A.fluid_in[pa + g1];
            const V4<float> b0 = A.fluid_in[pb + g0], b1 = A.fluid_in[pb + g1];
            const float2 fa = make_float2(A.field_in[pa + g0].x, A.field_in[pa + g1].x);
            const float2 fb = make_float2(A.field_in[pb + g0].x, A.field_in[pb + g1].x);
            q0 = recover_pair<FORM>(a0, a1, fa, P);
            recover_fix<FORM>(q0, &a0, &a1, fa, P);
            q1 = recover_pair<FORM>(b0, b1, fb, P);
            recover_fix<FORM>(q1, &b0, &b1, fb, P);
            phi_slot(z0 - 2)[pc] = fa;
            phi_slot(z0 - 1)[pc] = fb;
        }
        const int ix = cj * FXW + ci, iy = cj * 16 + ci;
        const bool v0 = ci < xe && cj < ye, v1 = ci < xe && cj + 8 < ye;
        if (!wait_raw(z0, true)) *dead = 1;
        plane_barrier();

        // phi of plane p beside the thread's pair, for the thermal form's faces
        auto phi_at = [&](int p, int d) {
            if constexpr (FORM == kThermal) return phi_slot(p)[pc + d];
            else return zero;
        };

        // One plane; the planes below z0 (ACT false) only fill the z pipeline.
        auto march = [&](int z, auto act) {
            constexpr bool ACT = decltype(act)::value;
            // phase A: recover plane z+2, face states, z flux
            const V4<float> *ru = raw_u + raw_slot(z + 2) * PC + rc;
            const V2<float> *rf = raw_f + raw_slot(z + 2) * PC + rc;
            float2 *wf = phi_slot(z + 2) + pc;
            P4 lox, loy;
            const float2 f2 = make_float2(rf[0].x, rf[8 * PW].x);
            P4 q2 = recover_pair<FORM>(ru[0], ru[8 * PW], f2, P);
            wf[0] = f2;
            if (cj == 0) wf[8 * PQ].x = f2.y;   // row 8 in pair row 8
            if (cj == 7) wf[-8 * PQ].y = f2.x;  // row 7 in pair row -1
            if constexpr (ACT) {
                P4 up;
                face_states_pair(get_pair<PP>(pr, pc - 1), q0, get_pair<PP>(pr, pc + 1), P.p_floor, lox, up);
                put_pair<FX>(hx, ix + 1, up);
                face_states_pair(get_pair<PP>(pr, pc - PQ), q0, get_pair<PP>(pr, pc + PQ), P.p_floor, loy, up);
                put_pair<FY>(hy, iy + 16, up);
                // the upper y state of row 7 is the lower side of face 8: second half of face pair 0
                if (cj == 7) put_half<FY, 0, 1>(hy, ci, up);
            }
            recover_fix<FORM>(q2, ru, ru + 8 * PW, f2, P);
            P4 fz_p;
            {
                P4 lo, up;
                face_states_pair(q0, q1, q2, P.p_floor, lo, up);
                FacePair f = face_pair(hiz, lo, phi_at(z, 0), phi_at(z + 1, 0));
                if (needs_clamp(f, zmax2)) clamp_face(f, zmax2);
                fz_p = hll_pair<2, FORM>(f, P);
                hiz = up;
            }
            plane_barrier();
            // phase B: publish plane z+1, x and y fluxes, load the combine's cells
            if (z + 4 <= zlast) issue(z + 4);
            put_pair<PP>(pr, pc, q1);
            if (cj == 0) put_half<PP, 1, 0>(pr, pc + 8 * PQ, q1);  // row 8 in pair row 8
            if (cj == 7) put_half<PP, 0, 1>(pr, pc - 8 * PQ, q1);  // row 7 in pair row -1
            V2<float> pf0, pf1, pn0, pn1;
            V4<float> pu0, pu1, un0, un1;
            P4 yl;
            const uint32_t base = (uint32_t)z * plane;
            if constexpr (ACT) {
                FacePair f = face_pair(get_pair<FX>(hx, ix), lox, phi_at(z, -1), phi_at(z, 0));
                if (needs_clamp(f, zmax2)) clamp_face(f, zmax2);
                put_pair<FX>(fx, ix, hll_pair<0, FORM>(f, P));
                // cells beyond the edge load their wrapped images and are not stored
                pf0 = A.field_in[base + g0];
                pf1 = A.field_in[base + g1];
                pu0 = A.fluid_in[base + g0];
                pu1 = A.fluid_in[base + g1];
                if (A.stage != 0) {
                    pn0 = A.field_n[base + g0];
                    pn1 = A.field_n[base + g1];
                    un0 = A.fluid_n[base + g0];
                    un1 = A.fluid_n[base + g1];
                }
                f = face_pair(get_pair<FY>(hy, iy), loy, phi_at(z, -PQ), phi_at(z, 0));
                if (needs_clamp(f, zmax2)) clamp_face(f, zmax2);
                yl = hll_pair<1, FORM>(f, P);
                put_pair<FY>(fy, iy, yl);
                if (cj == 0) put_half<FY, 1, 0>(fy, 8 * 16 + ci, yl);  // face 8 is also the first half of face pair 8
            }
            if (z + 3 <= zlast && !wait_raw(z + 3, z + 4 <= zlast)) *dead = 1;
            plane_barrier();
            // phase C: combine plane z (shaders/step.wgsl:149-173)
            if constexpr (ACT) {
                const float2 inv_dx = bc2(P.inv_dx), m2c = bc2(-2.0f);
                const float2 *fz = phi_slot(z) + pc;
                const float2 phi = fz[0];
                const float2 xm = fz[-1], xp = fz[1], ym = fz[-PQ], yp = fz[PQ];
                const float2 zm = phi_slot(z - 1)[pc], zp = phi_slot(z + 1)[pc];
                float2 lap = p_fma(m2c, phi, p_add(xm, xp));
                lap = p_add(lap, p_fma(m2c, phi, p_add(ym, yp)));
                lap = p_add(lap, p_fma(m2c, phi, p_add(zm, zp)));
                lap = p_mul(p_mul(lap, inv_dx), inv_dx);
                const float2 hdx = bc2(0.5f * P.inv_dx);
                const float2 gx = p_mul(p_sub(xp, xm), hdx), gy = p_mul(p_sub(yp, ym), hdx),
                             gz = p_mul(p_sub(zp, zm), hdx);
                const float2 pi = make_float2(pf0.y, pf1.y);
                const float2 om = p_sub(bc2(1.0f), dot3_2(q0.x, q0.y, q0.z));
                const float2 gam = make_float2(rsqrt_approx(fmaxf(om.x, 1e-12f)), rsqrt_approx(fmaxf(om.y, 1e-12f)));
                const float2 vg = p_fma(q0.z, gz, p_fma(q0.y, gy, p_mul(q0.x, gx)));
                const float2 drag = p_mul(bc2(P.eta), p_mul(gam, p_add(pi, vg)));
                float2 dpot = p_mul(phi, p_fma(p_fma(bc2(P.lambda), phi, bc2(-P.delta)), phi, bc2(P.m2)));
                float2 src = drag;
                if constexpr (FORM == kThermal) {
                    // the thermal part of dV/dphi, and its plasma part, exchanged like the friction
                    const float2 t = temperature_pair(q0.w, thermal_pair(phi, P), P);
                    const float2 dt = p_sub(t, bc2(P.t_ref));
                    const float2 gt = p_mul(bc2(P.th_g), p_mul(dt, p_add(t, bc2(P.t_ref))));
                    dpot = p_fma(phi, p_fma(p_mul(bc2(-P.th_a), dt), phi, gt), dpot);
                    src = p_fma(phi, p_fma(p_mul(bc2(-P.th_a), t), phi, p_mul(bc2(P.th_g), p_mul(t, t))), drag);
                }
                const float2 d_pi = p_sub(p_sub(lap, dpot), drag);
                // minus the flux divergence: ((dx + dy) + dz) / dx
                const P4 xl = get_pair<FX>(fx, ix), xu = get_pair<FX>(fx, ix + 1);
                const P4 yu = get_pair<FY>(fy, iy + 16);
                auto div = [&](float2 a, float2 b, float2 c, float2 d, float2 e, float2 f) {
                    return p_mul(p_add(p_add(p_sub(a, b), p_sub(c, d)), p_sub(e, f)), inv_dx);
                };
                const float2 nd = p_mul(src, bc2(-1.0f));
                const float2 d_e = p_fma(src, pi, div(xl.x, xu.x, yl.x, yu.x, fz_m.x, fz_p.x));
                const float2 d_x = p_fma(nd, gx, div(xl.y, xu.y, yl.y, yu.y, fz_m.y, fz_p.y));
                const float2 d_y = p_fma(nd, gy, div(xl.z, xu.z, yl.z, yu.z, fz_m.z, fz_p.z));
                const float2 d_z = p_fma(nd, gz, div(xl.w, xu.w, yl.w, yu.w, fz_m.w, fz_p.w));
                if (v0) store_cell<FORM>(A, base + g0, pf0, pu0, pn0, un0, d_pi.x, d_e.x, d_x.x, d_y.x, d_z.x, om.x);
                if (v1) store_cell<FORM>(A, base + g1, pf1, pu1, pn1, un1, d_pi.y, d_e.y, d_x.y, d_y.y, d_z.y, om.y);
            }
            q0 = q1;
            q1 = q2;
            fz_m = fz_p;
        };
        int z = z0 - 2;
#pragma unroll 1
        for (; z < z0 && !*dead; ++z) march(z, std::false_type{});
#pragma unroll 1
        for (; z >= z0 && z < z1 && !*dead; ++z) march(z, std::true_type{});
        stop = z;
    } else {
        // ---- halo warp -------------------------------------------------------------
        // h < 16: the upper x state of column -1 or the lower one of column 16 of
        // a row pair; else the upper y state of row -1 (first half) and the lower
        // one of row 16 (second half) of a column
        const bool xs = h < 16;
        P4 q1{}, s1{};  // the two ring pairs of plane z+1
        if (!wait_raw(z0, true)) *dead = 1;
        plane_barrier();
        int z = z0 - 2;
#pragma unroll 1
        for (; z < z1 && !*dead; ++z) {
            const bool act = z >= z0;
            const V4<float> *ru = raw_u + raw_slot(z + 2) * PC;
            const V2<float> *rf = raw_f + raw_slot(z + 2) * PC;
            float2 *wf = phi_slot(z + 2);
            const float2 f2 = make_float2(rf[rc].x, rf[rc + 8 * PW].x), f3 = make_float2(rf[r1a].x, rf[r1b].x);
            P4 q2 = recover_pair<FORM>(ru[rc], ru[rc + 8 * PW], f2, P);
            P4 s2 = recover_pair<FORM>(ru[r1a], ru[r1b], f3, P);
            wf[pc] = f2;
            wf[p1a].x = f3.x;
            wf[p1b].y = f3.y;
            if (act) {
                P4 a, b, c, lo, up;
                if (xs) {
                    const int at = (hj + 2) * PQ + (h < 8 ? 1 : 18);
                    a = get_pair<PP>(pr, at - 1);
                    b = get_pair<PP>(pr, at);
                    c = get_pair<PP>(pr, at + 1);
                } else {
                    const int at = (h & 15) + 2;
                    auto two = [&](int ra, int rb) {
                        const P4 u = get_pair<PP>(pr, ra * PQ + at), v = get_pair<PP>(pr, rb * PQ + at);
                        return P4{make_float2(u.x.x, v.x.y), make_float2(u.y.x, v.y.y), make_float2(u.z.x, v.z.y),
                                  make_float2(u.w.x, v.w.y)};
                    };
                    a = two(0, 9);   // rows -2 and 15
                    b = two(1, 10);  // rows -1 and 16
                    c = two(2, 11);  // rows 0 and 17
                }
                face_states_pair(a, b, c, P.p_floor, lo, up);
                if (h < 8) {
                    put_pair<FX>(hx, h * FXW, up);
                } else if (xs) {
                    put_pair<L::TY / 2>(lx, h - 8, lo);
                } else {
                    put_half<FY, 0, 0>(hy, h & 15, up);
                    ly[h & 15] = make_float4(lo.x.y, lo.y.y, lo.z.y, lo.w.y);
                }
            }
            recover_fix<FORM>(q2, ru + rc, ru + rc + 8 * PW, f2, P);
            recover_fix<FORM>(s2, ru + r1a, ru + r1b, f3, P);
            plane_barrier();
            if (z + 4 <= zlast) issue(z + 4);
            if (A.stage != 0 && z + kAhead >= z0 && z + kAhead < z1 && (h & 15) < ye) {
                // U^n of a later plane on its way to L2: two 128-byte lines of a row
                // of the fluid, one of the field
                const uint32_t row =
                    (uint32_t)(z + kAhead) * plane + (uint32_t)(y0 + (h & 15)) * (uint32_t)P.nx + (uint32_t)x0;
                if ((h >> 4) * 8 < xe) prefetch_l2(A.fluid_n + (row + (h >> 4) * 8));
                if (xs) prefetch_l2(A.field_n + row);
            }
            put_pair<PP>(pr, pc, q1);
            put_half<PP, 0, 0>(pr, p1a, s1);
            put_half<PP, 1, 1>(pr, p1b, s1);
            if (act && xs) {
                // h < 8: x face 16 of a row pair; else y face 16 of columns h - 8
                // and h, with x and y velocities (and momentum fluxes) exchanged so
                // one flux serves both
                P4 l, r;
                const bool xf = h < 8;
                const int i = h - 8;
                if (xf) {
                    l = get_pair<FX>(hx, h * FXW + 16);
                    r = get_pair<L::TY / 2>(lx, h);
                } else {
                    const P4 a = get_pair<FY>(hy, 8 * 16 + i), b = get_pair<FY>(hy, 8 * 16 + h);
                    l = P4{make_float2(a.y.y, b.y.y), make_float2(a.x.y, b.x.y), make_float2(a.z.y, b.z.y),
                           make_float2(a.w.y, b.w.y)};
                    const float4 c = ly[i], d = ly[h];
                    r = P4{make_float2(c.y, d.y), make_float2(c.x, d.x), make_float2(c.z, d.z), make_float2(c.w, d.w)};
                }
                float2 pl{}, pq{};
                if constexpr (FORM == kThermal) {
                    const float2 *fz = phi_slot(z);
                    if (xf) {  // columns 15 and 16
                        pl = fz[(h + 2) * PQ + 17];
                        pq = fz[(h + 2) * PQ + 18];
                    } else {  // rows 15 and 16 of the two columns
                        pl = make_float2(fz[9 * PQ + i + 2].y, fz[9 * PQ + h + 2].y);
                        pq = make_float2(fz[10 * PQ + i + 2].y, fz[10 * PQ + h + 2].y);
                    }
                }
                FacePair f = face_pair(l, r, pl, pq, !xf);
                if (needs_clamp(f, zmax2)) clamp_face(f, zmax2, !xf);
                P4 fl = hll_pair<0, FORM>(f, P);
                if (xf) {
                    put_pair<FX>(fx, h * FXW + 16, fl);
                } else {
                    const float2 m = fl.y;
                    fl.y = fl.z;
                    fl.z = m;
                    put_half<FY, 0, 1>(fy, 8 * 16 + i, fl);
                    put_half<FY, 1, 1>(fy, 8 * 16 + h, fl);
                }
            }
            if (z + 3 <= zlast && !wait_raw(z + 3, z + 4 <= zlast)) *dead = 1;
            plane_barrier();
            q1 = q2;
            s1 = s2;
        }
        stop = z;
    }
    if (stop == z1) return true;
    // The wait for plane stop + 2 expired: record it, wait (bounded) for the
    // copies in flight, stop.
    if (t == 0) {
        atomicOr(status, 1);
        if (tma) {
            wait_raw(stop + 2, false);
            if (stop + 3 <= zlast) wait_raw(stop + 3, false);
        }
    }
    return false;
}

template <int FORM>
__global__ void __launch_bounds__(PairLayout::NT, PairLayout::MIN_BLOCKS)
    pair_kernel(StageArgs<float> A, LatticeParams<float> P, int lz, const __grid_constant__ StageMaps maps, int tma_ok,
                int *status) {
    extern __shared__ __align__(128) unsigned char smem[];
    await_previous_launch();
    pair_item<FORM>(smem, A, P, lz, &maps, tma_ok, status, blockIdx.x, blockIdx.y);
}

}  // namespace dev
}  // namespace bubble
