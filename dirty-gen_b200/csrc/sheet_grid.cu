// Full-grid sheet substep for the coarse window and large grids.
//
// One substep of the reference (`substep`, x3-team/Dirty-gen
// src/fluid_core.rs:1879-2082) is split in two fused, tiled kernels:
//
//   k_force      eta = bed + h, the two 5-tap pressure blurs, gravity,
//                snapshot-Jacobi vorticity confinement, the divergence
//                "overload" projection (its own two blurs), damping and the
//                speed clamp. Reads h, bed, u, v (and grain/moisture for the
//                slurry), writes the new u, v. All intermediates live in
//                shared memory; the tile carries a 9-cell halo.
//   k_transport  donor-cell transport of depth, x pass then z pass, the dry
//                cut, and the FP64 ledger partial sum. Reads h, u, v, writes h.
//
// Both layers (water, slurry) go in one launch (blockIdx.z). Every stencil
// clamps its index at the grid edge exactly as the reference's edge branches
// do, so interior and border cells follow one formula.
//
// Work-box semantics: the reference steps only cells inside its work boxes
// (wet bounding box + 3, or split bodies + 6). A wet cell is always at least 3
// cells inside its box when a step has one substep, so every value a wet cell
// reads is a value the full-grid pass computes the same way; dry cells carry
// no flux and no force. The full-grid pass therefore gives the reference's
// depths and velocities on every cell that holds fluid.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <type_traits>
#include <vector>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include "sheet_grid.cuh"
#include "block_sum.cuh"
#include "sheet_math.cuh"
#include "launch_count.cuh"
#include "per_device.cuh"
#include "tile_geom.cuh"

namespace silt {

constexpr int FORCE_THREADS = 512;
constexpr int SNAP_CTAS = 3;  // per SM
constexpr size_t SWEEP_SMEM = 2 * Sweep::BYTES;  // a CTA's two teams
static_assert(2 * (SWEEP_SMEM + 2048) <= 228 * 1024, "two sweep CTAs share an SM");

// The threads that step one tile: a whole CTA, or one half of it (a barrier
// of its own). The sweep's time is block barriers between short stages (14.4
// barrier stalls per issue with two 512-thread tiles on an SM), which more
// and smaller teams fill for one another; with few tiles the latency of one
// tile counts, and a whole CTA takes it. A 1501^2 flood (2300 tile-layers):
// 376 us per launch by whole CTAs with a 9-cell halo, 348 by halves; 2048^2
// with a vehicle (360): 94 by whole CTAs, 129 by halves.
template <int N>
struct Team {
    static constexpr int NT = N;
    int tid, bar;
    __device__ Team() : tid((int)threadIdx.x % N), bar(N == FORCE_THREADS ? 0 : 1 + (int)threadIdx.x / N) {}
    __device__ __forceinline__ void sync() const {
        if constexpr (N == FORCE_THREADS)
            __syncthreads();
        else
            asm volatile("barrier.cta.sync %0, %1;" ::"r"(bar), "n"(N) : "memory");
    }
    __device__ __forceinline__ bool any(bool x) const {
        if constexpr (N == FORCE_THREADS) {
            return __syncthreads_or(x) != 0;
        } else {
            int r;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %1, 0;\n\tbarrier.cta.red.or.pred p, %2, %3, q;\n\t"
                "selp.s32 %0, 1, 0, p;\n\t}\n"
                : "=r"(r)
                : "r"((int)x), "r"(bar), "n"(N)
                : "memory");
            return r != 0;
        }
    }
};
using WholeCta = Team<FORCE_THREADS>;
using HalfCta = Team<FORCE_THREADS / 2>;

constexpr int TT = 32;       // transport tile edge
constexpr int TW = TT + 3;   // rows [t0-2, t1+1)
// A transport plane in shared memory: rows [ty0-2, ty0+33), each TS cells from
// column tx0-4 (16 bytes below tx0-2, so that a 2D TMA box can start there),
// padded to 128 bytes.
constexpr int TS = TT + 8;
constexpr int TPL = (TS * TW + 31) / 32 * 32;
static_assert((TS * sizeof(float)) % 16 == 0, "a TMA box row is a multiple of 16 bytes");
static_assert((TPL * sizeof(float)) % 128 == 0, "each transport plane starts 128-byte aligned");
static_assert(TS * TW * sizeof(float) <= TPL * sizeof(float), "a TMA box fits its plane");
constexpr int TRANSPORT_THREADS = 256;
// Per SM, by registers (six planes are 34 KB). The tile's six dependent stages
// wait at block barriers, which a fifth CTA fills: k_transport, whose grid is
// five per SM, 34 us with eight planes and four CTAs on a flooded 1000^2 grid
// and 31 so. The batch's grid is its tuner's choice, four per SM by default: six
// planes alone took it from 283 to 272 us on 256 windows.
constexpr int TRANSPORT_CTAS = 5;

size_t transport_smem_bytes() { return sizeof(float) * TPL * 6; }

// Five taps left to right. Away from the edge the reference starts from the
// first product (accum5); near it from 0.0 (accum5_clamped,
// src/fluid_core.rs:3680-3697).
__device__ __forceinline__ float tap5(float a0, float a1, float a2, float a3, float a4, float k0, float k1, float k2,
                                      bool interior) {
    float a = interior ? a0 * k0 : 0.0f + a0 * k0;
    a += a1 * k1;
    a += a2 * k2;
    a += a3 * k1;
    a += a4 * k0;
    return a;
}

__device__ __forceinline__ int clampi(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }

// The layer's substep count from its largest squared speed, in the host's
// arithmetic (IEEE sqrt and divide, no contraction).
__device__ __forceinline__ int device_nsub(const SubstepCount& c, int l) {
    const float m2 = __uint_as_float(c.speed2[l]);
    const float max_s = fmaxf(0.15f, sqrtf(m2));
    const float ns = ceilf((c.dt * max_s) / (0.42f * fmaxf(c.cell, 1.0e-3f)));
    return (int)rclamp(ns, 1.0f, c.cap);
}

// One flag plane by layer and buffer, without indexing the parameter array
// by a runtime value (which would copy it to local memory).
__device__ __forceinline__ uint8_t* pick(uint8_t* const (&a)[2][2], int l, int b) {
    return l ? (b ? a[1][1] : a[1][0]) : (b ? a[0][1] : a[0][0]);
}

// Tile-list entry: layer, zero-fill and copy bits over the tile index.
constexpr int ENTRY_ZERO = 1 << 29;
constexpr int ENTRY_COPY = 1 << 28;
constexpr int ENTRY_TILE = (1 << 28) - 1;

// Clears a sweep launch's barrier count and pass verdicts (the tile-list
// kernel does, before each force launch).
__device__ __forceinline__ void clear_sweep(SweepState* S) {
    if (!S) return;
    S->bar = 0u;
    S->flag[0] = S->flag[1] = S->flag[2] = 0u;
}

// Cell material: viscosity, mobility and damping factor.
__device__ __forceinline__ float cell_nu(const LayerParams& P, size_t g) {
    if (P.nu_mode == NU_CONST) return P.nu_c;
    if (P.nu_mode == NU_PLANE || P.nu_mode == NU_TABLE) return P.nu_plane[g];
    return dynamic_viscosity(P.grain[g], P.moisture[g]);
}

// sheet_mobility_for(nu) of the cell.
__device__ __forceinline__ float cell_mob(const LayerParams& P, size_t g) {
    if (P.nu_mode == NU_CONST) return P.mob_c;
    if (P.nu_mode == NU_TABLE) return P.mob_plane[g];
    return sheet_mobility_for(cell_nu(P, g));
}

// The cell's damping factor over dt: exp(-sheet_damp(nu) dt), the
// double-precision exponential rounded once (as the window engine does).
__device__ __forceinline__ float cell_decay(const LayerParams& P, size_t g, float dt) {
    if (P.nu_mode == NU_CONST) return P.decay_c;
    const float rate = P.nu_mode == NU_TABLE ? P.damp_plane[g] : sheet_damp(cell_nu(P, g));
    return exp_rn(-rate * dt);
}

// The damping factor of the viscosity a thread met last, for a layer with a
// viscosity plane (NU_PLANE; one such layer and one dt to a launch): a film of
// one material has one viscosity, and the factor is a double-precision power
// and exponential (k_force on a flooded 1000^2 grid of one viscosity 83 us
// evaluating it per cell, 70 so).
struct LastDamp {
    float nu = NAN, factor = 0.0f;  // NAN: none yet
    __device__ __forceinline__ float of(float x, float dt) {
        if (x != nu) {
            nu = x;
            factor = exp_rn(-sheet_damp(x) * dt);
        }
        return factor;
    }
};

// The velocity a substep starts from at (gx, gy), from the plane's (uu, vv):
// the lazy dry cut of the previous substep, then the soft window border
// (src/fluid_core.rs:9594-9622; a river reach's band keeps its current through
// the window ends). `band`: the border's width, 0 where no cell of the
// caller's tile lies in it (tile_band), which spares most tiles the distances.
__device__ __forceinline__ void start_velocity(const LayerParams& P, int band, int gx, int gy, float hv, float& uu,
                                               float& vv) {
    if (P.apply_cut && hv < P.eps) {
        uu = 0.0f;
        vv = 0.0f;
    }
    if (band > 0) {
        const int res = P.res;
        const int dx = min(gx, res - 1 - gx), dz = min(gy, res - 1 - gy);
        int d = min(dx, dz);
        if (P.open_axis == 1 && gy >= P.open_c0 && gy < P.open_c1) d = dz;
        else if (P.open_axis == 2 && gx >= P.open_c0 && gx < P.open_c1) d = dx;
        if (d < band) {
            float t = (float)d / (float)band;
            float w = t * t * (3.0f - 2.0f * t);
            uu *= w;
            vv *= w;
        }
    }
}

// P.soften_edge for a tile whose cells and halo reach the soft border, else 0.
template <class G>
__device__ __forceinline__ int tile_band(const LayerParams& P, int tx0, int ty0) {
    const int e = P.soften_edge + G::H;
    return min(tx0, ty0) < e || max(tx0, ty0) + FT + e > P.res ? P.soften_edge : 0;
}

// Shared-memory planes of a force tile (G::W x G::W floats each, origin at the
// tile corner minus G::H).
template <class G>
struct ForcePlanes {
    float* E;   // eta, then q
    float* TG;  // x-pass scratch; the snapshot form's vorticity between the two blurs
    float* TS;
    float* PB;  // pressure p, then projection b
    float* U;   // u, v
    float* V;
    float* HS;  // depth
    __device__ explicit ForcePlanes(float* sm)
        : E(sm), TG(sm + G::PLANE), TS(sm + 2 * G::PLANE), PB(sm + 3 * G::PLANE), U(sm + 4 * G::PLANE), V(sm + 5 * G::PLANE),
          HS(sm + 6 * G::PLANE) {}
};

#define NX(d) (EDGE ? (gy - oy) * G::W + (clampi(gx + (d), 0, res - 1) - ox) : s + (d))
#define NZ(d) (EDGE ? (clampi(gy + (d), 0, res - 1) - oy) * G::W + (gx - ox) : s + (d) * G::W)

// Tiles are staged by cp.async, one copy per value and plane, all of a stage
// in flight at once: a loop of loads and shared stores waits for each round
// trip in turn, since the compiler cannot move a load past a store through
// another pointer. (4-byte copies: rows start at any column.) A 1501^2 flood's
// sweep launch 305 -> 269 us, k_force on a flooded 1000^2 grid 100 -> 90, the
// transport there 39 -> 34.
__device__ __forceinline__ void stage(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
// Every thread's own copies have landed; a barrier publishes them to the team.
__device__ __forceinline__ void staged() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Depth and eta on radius R + 2, the velocity as stored on radius RV, then the
// pressure p = 0.45 (0.62 G + 0.38 S) + 0.55 eta on radius R (src/fluid_core.rs:1950-1985): the two 5-tap blurs,
// x pass then z pass. Ends with a barrier.
template <class TM, class G, bool EDGE, int R, int RV>
__device__ __forceinline__ void pressure_field(const TM& T, const LayerParams& P, const ForcePlanes<G>& F, int tx0,
                                               int ty0) {
    const int res = P.res;
    const int ox = tx0 - G::H, oy = ty0 - G::H;
    const float *depth = P.h, *bed = P.bed, *u = P.u, *v = P.v;
    region<TM, G, EDGE, R + 2, R + 2>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
        stage(&F.HS[s], depth + g);
        stage(&F.E[s], bed + g);
    });
    region<TM, G, EDGE, RV, RV>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
        stage(&F.U[s], u + g);
        stage(&F.V[s], v + g);
    });
    staged();
    region<TM, G, EDGE, R + 2, R + 2>(T, tx0, ty0, res, [&](int, int, int s, typename G::Index) { F.E[s] += F.HS[s]; });
    T.sync();
    region<TM, G, EDGE, R, R + 2>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
        const bool in = EDGE ? (gx >= 2 && gx <= res - 3) : true;
        float e0 = F.E[NX(-2)], e1 = F.E[NX(-1)], e2 = F.E[s], e3 = F.E[NX(1)], e4 = F.E[NX(2)];
        F.TG[s] = tap5(e0, e1, e2, e3, e4, kG0, kG1, kG2, in);
        F.TS[s] = tap5(e0, e1, e2, e3, e4, kS0, kS1, kS2, in);
    });
    T.sync();
    region<TM, G, EDGE, R, R>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
        const bool in = EDGE ? (gy >= 2 && gy <= res - 3) : true;
        const int s0 = NZ(-2), s1 = NZ(-1), s3 = NZ(1), s4 = NZ(2);
        float gb = tap5(F.TG[s0], F.TG[s1], F.TG[s], F.TG[s3], F.TG[s4], kG0, kG1, kG2, in);
        float sc = tap5(F.TS[s0], F.TS[s1], F.TS[s], F.TS[s3], F.TS[s4], kS0, kS1, kS2, in);
        float filtered = 0.62f * gb + 0.38f * sc;
        F.PB[s] = 0.45f * filtered + 0.55f * F.E[s];
    });
    T.sync();
}

// Projection, damping and the speed clamp from the confined velocity in U, V
// (radius 4), depth and eta (radius 4) (src/fluid_core.rs:1992-2037). Writes
// every cell of the tile to u_out, v_out.
template <class TM, class G, bool EDGE>
__device__ __forceinline__ void finish_tile(const TM& T, const LayerParams& P, const ForcePlanes<G>& F, int tx0, int ty0,
                                            LastDamp* last = nullptr) {
    const int res = P.res;
    const int ox = tx0 - G::H, oy = ty0 - G::H;
    const float dt = P.dt, eps = P.eps;
    if (P.project) {
        // b = div * overload - 0.015 * overload * lap(eta), radius 3 (:1992-2003).
        region<TM, G, EDGE, 3, 3>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
            const int sxp = NX(1), sxm = NX(-1), szp = NZ(1), szm = NZ(-1);
            float ux = fdiv(F.U[sxp] - F.U[sxm], P.div_two);
            float vz = fdiv(F.V[szp] - F.V[szm], P.div_two);
            float div = ux + vz;
            float lsum = F.E[sxp] + F.E[sxm] + F.E[szp] + F.E[szm] - 4.0f * F.E[s];
            float lap_h = fdiv(lsum, P.div_cell2);
            float overload = 1.0f + rclamp(fdiv(cell_nu(P, g), P.div_231), 0.0f, 6.0f);
            F.PB[s] = div * overload - 0.015f * overload * lap_h;
        });
        T.sync();
        // x pass of both blurs of b: rows radius 3, columns radius 1.
        region<TM, G, EDGE, 1, 3>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
            const bool in = EDGE ? (gx >= 2 && gx <= res - 3) : true;
            float b0 = F.PB[NX(-2)], b1 = F.PB[NX(-1)], b2 = F.PB[s], b3 = F.PB[NX(1)], b4 = F.PB[NX(2)];
            F.TG[s] = tap5(b0, b1, b2, b3, b4, kG0, kG1, kG2, in);
            F.TS[s] = tap5(b0, b1, b2, b3, b4, kS0, kS1, kS2, in);
        });
        T.sync();
        // q = 0.62 G(b) + 0.38 S(b), radius 1 (:2004-2011).
        region<TM, G, EDGE, 1, 1>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
            const bool in = EDGE ? (gy >= 2 && gy <= res - 3) : true;
            const int s0 = NZ(-2), s1 = NZ(-1), s3 = NZ(1), s4 = NZ(2);
            float gq = tap5(F.TG[s0], F.TG[s1], F.TG[s], F.TG[s3], F.TG[s4], kG0, kG1, kG2, in);
            float sq = tap5(F.TS[s0], F.TS[s1], F.TS[s], F.TS[s3], F.TS[s4], kS0, kS1, kS2, in);
            F.E[s] = 0.62f * gq + 0.38f * sq;
        });
        T.sync();
    }
    // Projection kick, damping and the speed clamp on wet cells (:2015-2037).
    region<TM, G, EDGE, 0, 0>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
        float uu = F.U[s], vv = F.V[s];
        if (F.HS[s] > eps) {
            if (P.project) {
                float qx = fdiv(F.E[NX(1)] - F.E[NX(-1)], P.div_two);
                float qz = fdiv(F.E[NZ(1)] - F.E[NZ(-1)], P.div_two);
                uu += 0.012f * dt * qx;
                vv += 0.012f * dt * qz;
            }
            float decay = last && P.nu_mode == NU_PLANE ? last->of(P.nu_plane[g], dt) : cell_decay(P, g, dt);
            uu = finite_speed(uu * decay, kSpeedCap);
            vv = finite_speed(vv * decay, kSpeedCap);
        }
        P.u_out[g] = uu;
        P.v_out[g] = vv;
    });
}

// One force tile in the snapshot (Jacobi) form. EDGE = false for tiles whose
// whole radius-9 region lies at least 2 cells inside the grid: no index is
// ever clamped there and every blur uses the interior form, so the stencils
// are plain offsets. Threads walk the regions as rows (one warp per row,
// lanes along x).
template <class TM, class G, bool EDGE>
__device__ __forceinline__ void force_tile(const TM& T, const LayerParams& P, float* sm, int tx0, int ty0,
                                           LastDamp* last) {
    const int res = P.res;
    const ForcePlanes<G> F(sm);
    const int ox = tx0 - G::H, oy = ty0 - G::H;
    const int band = tile_band<G>(P, tx0, ty0);
    const float dt = P.dt, eps = P.eps;
    // 1-3. Depth, eta (radius 9) and the pressure (radius 7).
    pressure_field<TM, G, EDGE, 7, 6>(T, P, F, tx0, ty0);
    // Velocity on radius 6 and gravity down the pressure gradient on wet
    // cells (src/fluid_core.rs:2234-2253).
    region<TM, G, EDGE, 6, 6>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
        float uu = F.U[s], vv = F.V[s];
        start_velocity(P, band, gx, gy, F.HS[s], uu, vv);
        if (F.HS[s] > eps) {
            float px = fdiv(F.PB[NX(1)] - F.PB[NX(-1)], P.div_two);
            float pz = fdiv(F.PB[NZ(1)] - F.PB[NZ(-1)], P.div_two);
            float mob = cell_mob(P, g);
            uu += -kGravity * px * mob * dt;
            vv += -kGravity * pz * mob * dt;
        }
        F.U[s] = uu;
        F.V[s] = vv;
    });
    T.sync();
    // Vorticity of the post-gravity snapshot, radius 5 (src/fluid_core.rs:3498-3506).
    if (P.vort > 0.0f) {
        region<TM, G, EDGE, 5, 5>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
            float dvdx = fdiv(F.V[NX(1)] - F.V[NX(-1)], P.div_two);
            float dudz = fdiv(F.U[NZ(1)] - F.U[NZ(-1)], P.div_two);
            F.TG[s] = dvdx - dudz;
        });
        T.sync();
        // Confinement kick from that snapshot, in place, radius 4
        // (src/fluid_core.rs:2348-2375, :2441-2470).
        region<TM, G, EDGE, 4, 4>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
            if (F.HS[s] > eps) {
                float w = F.TG[s];
                if (finite_f(w) && !(fabsf(w) < 1.0e-4f)) {
                    float wxp = fabsf(F.TG[NX(1)]), wxm = fabsf(F.TG[NX(-1)]);
                    float wzp = fabsf(F.TG[NZ(1)]), wzm = fabsf(F.TG[NZ(-1)]);
                    float nx_ = fdiv(wxp - wxm, P.div_two);
                    float nz_ = fdiv(wzp - wzm, P.div_two);
                    float du = P.vort * dt * (-nz_ * w);
                    float dv = P.vort * dt * (nx_ * w);
                    if (finite_f(du) && finite_f(dv) && du * du + dv * dv <= 0.0625f) {
                        F.U[s] += du;
                        F.V[s] += dv;
                    }
                }
            }
        });
        T.sync();
    }
    finish_tile<TM, G, EDGE>(T, P, F, tx0, ty0, last);
}

// Sweep form, part 1: the post-gravity velocity G of every cell of the tile
// (gravity on wet cells only; a dry cell keeps its starting velocity), written
// to u_out, v_out, and the sweep's first iterate F = G to fu, fv.
template <class TM, class G, bool EDGE>
__device__ __forceinline__ void pre_tile(const TM& T, const LayerParams& P, float* sm, int tx0, int ty0) {
    const int res = P.res;
    const ForcePlanes<G> F(sm);
    const int ox = tx0 - G::H, oy = ty0 - G::H;
    const int band = tile_band<G>(P, tx0, ty0);
    const float dt = P.dt, eps = P.eps;
    pressure_field<TM, G, EDGE, 1, 0>(T, P, F, tx0, ty0);
    region<TM, G, EDGE, 0, 0>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
        float uu = F.U[s], vv = F.V[s];
        start_velocity(P, band, gx, gy, F.HS[s], uu, vv);
        if (F.HS[s] > eps) {
            float px = fdiv(F.PB[NX(1)] - F.PB[NX(-1)], P.div_two);
            float pz = fdiv(F.PB[NZ(1)] - F.PB[NZ(-1)], P.div_two);
            float mob = cell_mob(P, g);
            uu += -kGravity * px * mob * dt;
            vv += -kGravity * pz * mob * dt;
        }
        P.u_out[g] = uu;
        P.v_out[g] = vv;
        P.fu[g] = uu;
        P.fv[g] = vv;
    });
}

// Sweep form, part 2: one pass of the raster-order Gauss-Seidel confinement
// (force_gravity_open, src/fluid_core.rs:2234-2260) solved as a fixed point.
// In the reference's sweep a wet cell's final velocity is its post-gravity
// value G plus the kick computed from the final values of the cells before it
// in raster order, its own G, and the starting values of the cells after it;
// dry cells never change. The tile iterates that equation for its own wet
// cells in shared memory, reading the current iterate of other tiles' cells
// from fu, fv, until a local pass changes no bit (each pass settles at least
// the first unsettled cell in raster order, so it ends), and writes back what
// changed. Returns true (block-uniform) when a value another tile reads
// changed. When a whole pass over every tile changes none, every cell
// satisfies its equation with the values it read, and since each cell depends
// only on earlier cells that solution is the sequential sweep's, bit for bit.
//
// A change at c reaches the cells that read c's iterate: c + (1,0), (2,0),
// (0,1), (-1,1), (1,1), (0,2) (index clamping at the grid's edge reads no
// other cells). So a local pass after the first recomputes only the marked
// ones; the first pass of a tile solved before (`again`) only those that read
// the ring of other tiles' cells, the 154 of rows 0-1 and columns 0, 1 and
// 31, since the tile's own values satisfy their equations; and only a change
// in column 0, 30 or 31 or in row 30 or 31 is another tile's business.
// Recomputing whole tiles in every pass, a flood's launch of 2300 tile-layers
// (2.5 solves each) took 348 us instead of 305.
// `reuse`: this team's shared memory still holds this tile from an earlier
// pass of the launch (the team solves no other tile), so only the ring of
// other tiles' wet cells around it is read again; the starting and
// post-gravity velocities and the tile's own iterate are current.
template <class TM, class G, bool EDGE>
__device__ bool sweep_tile(const TM& T, const LayerParams& P, float* sm, int tx0, int ty0, bool again, bool reuse,
                           int& passes) {
    const int res = P.res;
    float* PU = sm;              // starting velocity (the values of cells after a cell)
    float* PV = sm + G::PLANE;
    float* FU = sm + 2 * G::PLANE;  // current iterate (the values of cells before it)
    float* FV = sm + 3 * G::PLANE;
    float* GU = sm + 4 * G::PLANE;  // post-gravity velocity of the tile's own cells
    float* GV = sm + 5 * G::PLANE;
    float* HS = sm + 6 * G::PLANE;  // depth
    // Marks of the cells to recompute: pass it reads one byte plane, clearing
    // it, and marks in the other; both are clear when a solve ends.
    uint8_t* const marks = reinterpret_cast<uint8_t*>(sm + 7 * G::PLANE);
    const int ox = tx0 - G::H, oy = ty0 - G::H;
    const int band = tile_band<G>(P, tx0, ty0);
    const float eps = P.eps, dt = P.dt, vort = P.vort;
    const FixedDiv two = P.div_two;
    float *__restrict__ fu = P.fu, *__restrict__ fv = P.fv;
    auto own = [&](int gx, int gy) { return gx >= tx0 && gx < tx0 + FT && gy >= ty0 && gy < ty0 + FT; };
    if (reuse) {
        region<TM, G, EDGE, 2, 2>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
            if (!own(gx, gy) && HS[s] > eps) {
                stage(&FU[s], fu + g);
                stage(&FV[s], fv + g);
            }
        });
        staged();
    } else {
        const float *depth = P.h, *u = P.u, *v = P.v, *gu = P.u_out, *gv = P.v_out;
        region<TM, G, EDGE, 2, 2>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
            stage(&HS[s], depth + g);
            stage(&PU[s], u + g);
            stage(&PV[s], v + g);
            stage(&FU[s], fu + g);
            stage(&FV[s], fv + g);
            if (own(gx, gy)) {
                stage(&GU[s], gu + g);
                stage(&GV[s], gv + g);
                marks[s] = marks[G::PLANE + s] = 0;
            }
        });
        staged();
        // The same thread's cells again.
        region<TM, G, EDGE, 2, 2>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index) {
            const float hv = HS[s];
            float uu = PU[s], vv = PV[s];
            start_velocity(P, band, gx, gy, hv, uu, vv);
            PU[s] = uu;
            PV[s] = vv;
            // A wet cell's tile is always stepped this substep, so its iterate
            // is current; a dry cell keeps its starting velocity.
            if (!(hv > eps)) {
                FU[s] = uu;
                FV[s] = vv;
            }
        });
    }
    T.sync();
    bool exported = false;
    int changed = 0;
    uint8_t* mark_next = nullptr;
    auto solve = [&](int gx, int gy, int s) {
        float du, dv, nu_ = GU[s], nv_ = GV[s];
        int kick = -1;
        if (!EDGE || (gx >= 2 && gy >= 2 && gx < res - 2 && gy < res - 2))
            kick = conf_kick_inner<false>(two, dt, vort, SweepRead{FU, PU, GU, s, G::W}, SweepRead{FV, PV, GV, s, G::W}, du,
                                   dv);
        if (kick < 0) {
            auto at = [&](int a, int b) { return (b - oy) * G::W + (a - ox); };
            auto before = [&](int a, int b) { return b < gy || (b == gy && a < gx); };
            auto uu = [&](int a, int b) {
                if (a == gx && b == gy) return GU[s];
                return before(a, b) ? FU[at(a, b)] : PU[at(a, b)];
            };
            auto vv = [&](int a, int b) {
                if (a == gx && b == gy) return GV[s];
                return before(a, b) ? FV[at(a, b)] : PV[at(a, b)];
            };
            kick = conf_kick(gx, gy, res, two, dt, vort, uu, vv, du, dv);
        }
        if (kick) {
            nu_ = GU[s] + du;
            nv_ = GV[s] + dv;
        }
        if (__float_as_uint(nu_) != __float_as_uint(FU[s]) || __float_as_uint(nv_) != __float_as_uint(FV[s])) {
            FU[s] = nu_;
            FV[s] = nv_;
            changed |= (gx == tx0 || gx >= tx0 + FT - 2 || gy >= ty0 + FT - 2) ? 3 : 1;
            mark_next[s + 1] = 1;
            mark_next[s + 2] = 1;
            mark_next[s + G::W - 1] = 1;
            mark_next[s + G::W] = 1;
            mark_next[s + G::W + 1] = 1;
            mark_next[s + 2 * G::W] = 1;
        }
    };
    bool tile_changed = false;
    passes = 0;
    for (int it = 0; it <= FT * FT; ++it) {
        ++passes;
        changed = 0;
        uint8_t* const mark = marks + (it & 1) * G::PLANE;
        mark_next = marks + ((it + 1) & 1) * G::PLANE;
        if (it == 0 && again) {
            constexpr int N = 2 * FT + 3 * (FT - 2);
            for (int k = T.tid; k < N; k += TM::NT) {
                const int q = k - 2 * FT, c = q % 3;
                const int gx = tx0 + (q < 0 ? k % FT : (c == 2 ? FT - 1 : c)), gy = ty0 + (q < 0 ? k / FT : 2 + q / 3);
                if (EDGE && (gx >= res || gy >= res)) continue;
                const int s = (gy - oy) * G::W + (gx - ox);
                if (HS[s] > eps) solve(gx, gy, s);
            }
        } else {
            region<TM, G, EDGE, 0, 0>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index) {
                if (it > 0) {
                    if (!mark[s]) return;
                    mark[s] = 0;
                }
                if (HS[s] > eps) solve(gx, gy, s);
            });
        }
        exported |= (changed & 2) != 0;
        if (!T.any(changed != 0)) break;
        tile_changed = true;
    }
    if (tile_changed) {
        region<TM, G, EDGE, 0, 0>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index g) {
            if (HS[s] > eps) {
                fu[g] = FU[s];
                fv[g] = FV[s];
            }
        });
    }
    return T.any(exported);  // and shared memory is read again by the next tile or pass
}

// Sweep form, part 3: projection, damping and clamp from the solved sweep.
template <class TM, class G, bool EDGE>
__device__ __forceinline__ void post_tile(const TM& T, const LayerParams& P, float* sm, int tx0, int ty0) {
    const int res = P.res;
    const ForcePlanes<G> F(sm);
    const int band = tile_band<G>(P, tx0, ty0);
    const float eps = P.eps;
    const float *depth = P.h, *bed = P.bed, *u = P.u, *v = P.v, *fu = P.fu, *fv = P.fv;
    region<TM, G, EDGE, 4, 4>(T, tx0, ty0, res, [&](int, int, int s, typename G::Index g) {
        stage(&F.HS[s], depth + g);
        stage(&F.E[s], bed + g);
        stage(&F.U[s], u + g);
        stage(&F.V[s], v + g);
        stage(&F.TG[s], fu + g);
        stage(&F.TS[s], fv + g);
    });
    staged();
    region<TM, G, EDGE, 4, 4>(T, tx0, ty0, res, [&](int gx, int gy, int s, typename G::Index) {
        const float hv = F.HS[s];
        F.E[s] += hv;
        float uu = F.U[s], vv = F.V[s];
        if (hv > eps) {
            uu = F.TG[s];
            vv = F.TS[s];
        } else {
            start_velocity(P, band, gx, gy, hv, uu, vv);
        }
        F.U[s] = uu;
        F.V[s] = vv;
    });
    T.sync();
    finish_tile<TM, G, EDGE>(T, P, F, tx0, ty0);
}

#undef NX
#undef NZ

// A layer's force parameters for this substep: with a device count, its dt
// and (constant-viscosity layers) damping factor for that count.
__device__ __forceinline__ LayerParams force_params(const LayerParams& P0, const SubstepCount& sc, int l,
                                                    bool report_overflow) {
    LayerParams P = P0;
    if (sc.speed2) {
        const int ns = device_nsub(sc, l);
        P.dt = sc.dt / (float)ns;
        if (P.nu_mode == NU_CONST) P.decay_c = sc.water_decay[ns];
        if (report_overflow && sc.k == 0 && ns > sc.launched) atomicOr(sc.overflow, 1u);
    }
    return P;
}

// A tile whose whole region lies at least 2 cells inside the grid: no stencil
// index is clamped there and every blur uses the interior form.
template <class G>
__device__ __forceinline__ bool tile_interior(int res, int tx0, int ty0) {
    return tx0 - G::H >= 2 && ty0 - G::H >= 2 && tx0 + FT + G::H <= res - 2 && ty0 + FT + G::H <= res - 2;
}

// One list entry of the force pass (the sweep form's first part for a
// sweeping layer). Returns true when it used shared memory.
template <class G, class TM>
__device__ __forceinline__ bool force_entry(const TM& T, const LayerParams& P, const TileFlags& tf, int nxt, int e, float* sm,
                                            LastDamp* last = nullptr) {
    const int l = e >> 30, zero_fill = (e & ENTRY_ZERO) != 0, copy = (e & ENTRY_COPY) != 0, t = e & ENTRY_TILE;
    const int res = P.res;
    const int tx0 = (t % tf.tiles_x) * FT, ty0 = (t / tf.tiles_x) * FT;
    if (copy) {
        // Identity substep of a layer that has taken all its substeps.
        const int w = min(FT, res - tx0), h = min(FT, res - ty0);
        for (int q = T.tid; q < w * h; q += TM::NT) {
            const size_t g = (size_t)(ty0 + q / w) * res + tx0 + q % w;
            P.u_out[g] = P.u[g];
            P.v_out[g] = P.v[g];
        }
        if (T.tid == 0) pick(tf.zero_uv, l, nxt)[t] = pick(tf.zero_uv, l, nxt ^ 1)[t];
        return false;
    }
    if (zero_fill) {
        // A quiet tile: dry in its whole neighbourhood, so after the dry cut
        // its velocity is zero.
        const int w = min(FT, res - tx0), h = min(FT, res - ty0);
        for (int q = T.tid; q < w * h; q += TM::NT) {
            const size_t g = (size_t)(ty0 + q / w) * res + tx0 + q % w;
            P.u_out[g] = 0.0f;
            P.v_out[g] = 0.0f;
        }
        if (T.tid == 0) pick(tf.zero_uv, l, nxt)[t] = 1;
        return false;
    }
    const bool interior = tile_interior<G>(res, tx0, ty0);
    if constexpr (std::is_same_v<G, Sweep>) {
        // Sweep form: this launch's first part; the sweep and the projection follow.
        if (interior)
            pre_tile<TM, G, false>(T, P, sm, tx0, ty0);
        else
            pre_tile<TM, G, true>(T, P, sm, tx0, ty0);
    } else if (interior) {
        force_tile<TM, G, false>(T, P, sm, tx0, ty0, last);
    } else {
        force_tile<TM, G, true>(T, P, sm, tx0, ty0, last);
    }
    if (T.tid == 0) pick(tf.zero_uv, l, nxt)[t] = 0;
    return true;
}

// A list entry that steps its tile (neither a zero fill nor an identity copy).
__device__ __forceinline__ bool entry_steps(int e) { return (e & (ENTRY_ZERO | ENTRY_COPY)) == 0; }

// Sweep-form pass `pass` over one list entry: the fixed-point pass of a
// stepped tile of a sweeping layer with confinement on. After the first
// pass a tile is solved again only when a tile whose cells it reads as
// earlier ones (left, right and the three above) changed since the previous
// pass began: it is otherwise still at the fixed point of the values around
// it. Returns whether a value another tile reads changed (block-uniform) and
// stamps the tile when one did. `reuse`: the team solves only this entry in
// the launch, so its shared memory keeps the tile between passes.
template <class TM>
__device__ __forceinline__ bool sweep_entry(const TM& T, const LayerParams& P, const TileFlags& tf, int e, float* sm,
                                            int pass, unsigned int epoch, bool reuse) {
    if (!entry_steps(e) || !P.sweep || !(P.vort > 0.0f)) return false;
    const int l = e >> 30, t = e & ENTRY_TILE;
    const int nt = tf.tiles_x * tf.tiles_x;
    const int ti = t % tf.tiles_x, tj = t / tf.tiles_x;
    unsigned int* stamp = tf.stamp + (size_t)l * nt;
    if (pass > 0) {
        // Five threads read the five stamps at once.
        bool hit = false;
        if (T.tid < 5) {
            const int x = ti + (T.tid < 3 ? T.tid - 1 : 2 * T.tid - 7), y = tj - (T.tid < 3 ? 1 : 0);
            const unsigned int since = epoch * 256u + (unsigned int)pass;
            hit = x >= 0 && y >= 0 && x < tf.tiles_x &&
                  *(volatile unsigned int*)&stamp[y * tf.tiles_x + x] >= since;
        }
        if (!T.any(hit)) return false;
    }
    const int tx0 = ti * FT, ty0 = tj * FT;
    int passes = 0;
    const bool again = pass > 0, keep = reuse && again;
    const bool changed = tile_interior<Sweep>(P.res, tx0, ty0)
                             ? sweep_tile<TM, Sweep, false>(T, P, sm, tx0, ty0, again, keep, passes)
                             : sweep_tile<TM, Sweep, true>(T, P, sm, tx0, ty0, again, keep, passes);
    if (T.tid == 0) {
        if (changed) {
            __threadfence();
            stamp[t] = epoch * 256u + (unsigned int)pass + 1u;
        }
        if (tf.sweep) {
            atomicAdd(&tf.sweep->solves, 1u);
            atomicAdd(&tf.sweep->local_passes, (unsigned int)passes);
        }
    }
    return changed;
}

// Sweep-form projection of one list entry. Returns true when it used shared memory.
template <class TM>
__device__ __forceinline__ bool post_entry(const TM& T, const LayerParams& P, const TileFlags& tf, int e, float* sm) {
    if (!entry_steps(e) || !P.sweep) return false;
    const int t = e & ENTRY_TILE;
    const int tx0 = (t % tf.tiles_x) * FT, ty0 = (t / tf.tiles_x) * FT;
    if (tile_interior<Sweep>(P.res, tx0, ty0))
        post_tile<TM, Sweep, false>(T, P, sm, tx0, ty0);
    else
        post_tile<TM, Sweep, true>(T, P, sm, tx0, ty0);
    return true;
}

// ----------------------------------------------- Gauss-Seidel sweep launches
//
// The sweep's fixed point couples every stepped tile, so its passes run in
// one cooperative launch (every CTA resident at once) separated by a grid
// barrier. Each wait is bounded: past the limit the CTA records the failure
// in SweepState::err and the launch ends; the host reports SILT_ETIMEOUT.

constexpr int SWEEP_MAX_PASSES = 64;                  // then the sequential sweep
constexpr unsigned int SWEEP_SPIN_LIMIT = 1u << 22;   // polls of ~0.1 us: about half a second

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid barrier of a cooperative launch: the arrival count only grows within
// a launch (the tile-list kernel clears it before), so barrier number k waits
// for k * gridDim.x arrivals. False when the wait gave up.
__device__ bool grid_barrier(SweepState* S, unsigned int& target) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        __threadfence();
        atomicAdd(&S->bar, 1u);
        int good = 1;
        unsigned int spins = 0;
        while (ld_acquire_u32(&S->bar) < target) {
            if (++spins > SWEEP_SPIN_LIMIT) {
                atomicOr(&S->err, 1u);
                good = 0;
                break;
            }
            if (spins > 256) __nanosleep(64);  // short waits poll without sleeping
        }
        __threadfence();
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// A team's share of a launch over its list: the first entry it takes, the
// step to its next, its shared memory and its half of the CTA.
template <class TM>
struct SweepTeam {
    TM T;
    int half, first, stride;
    float* sm;
    __device__ explicit SweepTeam(float* shared) {
        constexpr int TEAMS = FORCE_THREADS / TM::NT;
        half = (int)threadIdx.x / TM::NT;
        first = (int)blockIdx.x + half * (int)gridDim.x;
        stride = TEAMS * (int)gridDim.x;
        sm = shared + half * (Sweep::BYTES / sizeof(float));
    }
};

// Passes of the fixed point until one changes nothing anywhere. `visit(k)`
// runs list entry k's pass and returns whether it changed a value. Returns
// the number of passes, 0 at the pass limit, -1 after a failed barrier.
template <class TM, class Visit>
__device__ int sweep_fixed_point(const SweepTeam<TM>& W, SweepState* S, unsigned int& target, int n, Visit visit) {
    __shared__ unsigned int verdict;
    for (int pass = 0; pass < SWEEP_MAX_PASSES; ++pass) {
        bool changed = false;
        for (int k = W.first; k < n; k += W.stride) changed |= visit(k, pass);
        if (W.T.tid == 0 && changed) atomicOr(&S->flag[pass % 3], 1u);
        // The next pass's verdict starts clear; the one cleared here was
        // last read before the previous barrier.
        if (threadIdx.x == 0 && blockIdx.x == 0) S->flag[(pass + 1) % 3] = 0u;
        if (!grid_barrier(S, target)) return -1;
        if (threadIdx.x == 0) verdict = ld_acquire_u32(&S->flag[pass % 3]);
        __syncthreads();
        if (verdict == 0u) return pass + 1;
    }
    return 0;
}

// The sequential sweep of one layer on one thread (past the pass limit):
// every wet cell in raster order, as force_gravity_open does.
__device__ void sweep_serial(const LayerParams& P) {
    const int res = P.res;
    const float eps = P.eps;
    for (int j = 0; j < res; ++j)
        for (int i = 0; i < res; ++i) {
            const size_t g = (size_t)j * res + i;
            if (!(P.h[g] > eps)) continue;
            auto val = [&](bool is_u, int a, int b) {
                const size_t q = (size_t)b * res + a;
                if (a == i && b == j) return is_u ? P.u_out[q] : P.v_out[q];
                const float hq = P.h[q];
                if (hq > eps && (b < j || (b == j && a < i))) return is_u ? P.fu[q] : P.fv[q];
                float uu = P.u[q], vv = P.v[q];
                start_velocity(P, P.soften_edge, a, b, hq, uu, vv);
                return is_u ? uu : vv;
            };
            auto uu = [&](int a, int b) { return val(true, a, b); };
            auto vv = [&](int a, int b) { return val(false, a, b); };
            float du, dv, nu_ = P.u_out[g], nv_ = P.v_out[g];
            if (conf_kick(i, j, res, P.div_two, P.dt, P.vort, uu, vv, du, dv)) {
                nu_ = P.u_out[g] + du;
                nv_ = P.v_out[g] + dv;
            }
            P.fu[g] = nu_;
            P.fv[g] = nv_;
        }
}

// True when layer l takes a real (not identity) substep in this launch.
__device__ __forceinline__ bool layer_steps(const SubstepCount& sc, int l) {
    return !(sc.speed2 && sc.k > 0 && sc.k >= device_nsub(sc, l));
}

__device__ __forceinline__ void sweep_stats(SweepState* S, int passes) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&S->launches, 1u);
        atomicAdd(&S->epoch, 1u);  // every CTA read the epoch at the launch's start, two barriers ago
        atomicMax(&S->passes_max, (unsigned int)(passes > 0 ? passes : SWEEP_MAX_PASSES));
        if (passes == 0) atomicAdd(&S->fallbacks, 1u);
    }
}

// One sheet's force pass in the sweep form: pre-sweep tiles (and the list's
// zero and copy entries), the fixed point, projection.
template <class TM>
__device__ __forceinline__ void force_sweep(const ForceLaunch& L, const LayerParams* Ps, int n, float* sm) {
    SweepState* S = L.tf.sweep;
    const unsigned int epoch = ld_acquire_u32(&S->epoch);
    const SweepTeam<TM> W(sm);
    for (int k = W.first; k < n; k += W.stride) {
        const int e = L.tf.list[k];
        if (force_entry<Sweep>(W.T, Ps[e >> 30], L.tf, L.nxt, e, W.sm)) W.T.sync();
    }
    unsigned int target = 0;
    if (!grid_barrier(S, target)) return;
    const bool reuse = n <= W.stride;  // one entry per team: its tile stays in shared memory
    const int passes = sweep_fixed_point(W, S, target, n, [&](int k, int pass) {
        const int e = L.tf.list[k];
        return sweep_entry(W.T, Ps[e >> 30], L.tf, e, W.sm, pass, epoch, reuse);
    });
    if (passes < 0) return;
    if (passes == 0) {
        if (threadIdx.x == 0 && blockIdx.x < 2) {
            const LayerParams& P = Ps[blockIdx.x];
            if (P.sweep && P.vort > 0.0f && !P.skip && layer_steps(L.sc, blockIdx.x)) sweep_serial(P);
        }
        if (!grid_barrier(S, target)) return;
    }
    sweep_stats(S, passes);
    for (int k = W.first; k < n; k += W.stride) {
        const int e = L.tf.list[k];
        if (post_entry(W.T, Ps[e >> 30], L.tf, e, W.sm)) W.T.sync();
    }
}

// force_sweep as a cooperative launch; its teams are whole CTAs while every
// entry of the list has one.
__global__ void __launch_bounds__(FORCE_THREADS, 2) k_force_sweep(ForceLaunch L) {
    ::silt::dep_wait();
    extern __shared__ float sm[];
    __shared__ LayerParams Ps[2];
    if (threadIdx.x < 2) Ps[threadIdx.x] = force_params(L.lay[threadIdx.x], L.sc, threadIdx.x, blockIdx.x == 0);
    __syncthreads();
    const int n = *L.tf.count;
    if (n <= (int)gridDim.x)
        force_sweep<WholeCta>(L, Ps, n, sm);
    else
        force_sweep<HalfCta>(L, Ps, n, sm);
}

// The snapshot form's force pass, persistent over the substep's tile list.
template <class G>
__device__ __forceinline__ void force_snapshot(const ForceLaunch& L) {
    extern __shared__ float sm[];
    __shared__ LayerParams Ps[2];
    if (threadIdx.x < 2) Ps[threadIdx.x] = force_params(L.lay[threadIdx.x], L.sc, threadIdx.x, blockIdx.x == 0);
    __syncthreads();
    const int n = *L.tf.count;
    const WholeCta T;
    LastDamp last;
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const int e = L.tf.list[k];
        if (force_entry<G>(T, Ps[e >> 30], L.tf, L.nxt, e, sm, &last)) T.sync();  // shared memory is reused by the next tile
    }
}

__global__ void __launch_bounds__(FORCE_THREADS, SNAP_CTAS) k_force(ForceLaunch L) {
    ::silt::dep_wait();
    force_snapshot<Snap>(L);
}

// On a grid of more than MAX_NEAR_RES cells a side.
__global__ void __launch_bounds__(FORCE_THREADS, SNAP_CTAS) k_force_far(ForceLaunch L) {
    ::silt::dep_wait();
    force_snapshot<FarSnap>(L);
}

// The list entry of tile t of layer l for this substep, or -1 for none.
__device__ __forceinline__ int tile_entry(const TileFlags& tf, int cur, int nxt, int all, const SubstepCount& sc,
                                          int l, int t) {
    if (sc.speed2 && sc.k > 0) {  // substep 0 steps every layer; its list precedes the speed pass
        const int ns = device_nsub(sc, l);
        if (sc.k >= ns) {
            // Identity substep: carry every tile not known to be zero.
            if (!(pick(tf.zero_h, l, cur)[t] && pick(tf.zero_uv, l, cur)[t])) return (l << 30) | ENTRY_COPY | t;
            if (!(pick(tf.zero_h, l, nxt)[t] && pick(tf.zero_uv, l, nxt)[t])) return (l << 30) | ENTRY_ZERO | t;
            return -1;
        }
    }
    const int ti = t % tf.tiles_x, tj = t / tf.tiles_x;
    bool active = all != 0;
    for (int dj = -1; dj <= 1 && !active; ++dj)
        for (int di = -1; di <= 1; ++di) {
            const int a = ti + di, b = tj + dj;
            if (a < 0 || b < 0 || a >= tf.tiles_x || b >= tf.tiles_x) continue;
            if (pick(tf.wet, l, cur)[b * tf.tiles_x + a]) {
                active = true;
                break;
            }
        }
    if (active) {
        if (tf.stepped) atomicAdd(&tf.stepped[l], 1ull);
        return (l << 30) | t;
    }
    if (!pick(tf.zero_uv, l, nxt)[t] || !pick(tf.zero_h, l, nxt)[t]) return (l << 30) | ENTRY_ZERO | t;
    return -1;
}

__global__ void k_tile_list(TileFlags tf, int cur, int nxt, int all, int skip0, int skip1, SubstepCount sc,
                            int* count_next, double* zero_ledger, unsigned int* zero_bits, const double* sum,
                            double wet) {
    ::silt::dep_wait();
    const int nt = tf.tiles_x * tf.tiles_x;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (sum && !(*sum > wet)) return;
    if (k == 0) {
        if (count_next) *count_next = 0;
        if (zero_ledger) zero_ledger[0] = zero_ledger[1] = 0.0;
        if (zero_bits) zero_bits[0] = zero_bits[1] = 0u;
        clear_sweep(tf.sweep);
    }
    if (k >= 2 * nt) return;
    const int l = k / nt, t = k % nt;
    if (l == 0 ? skip0 : skip1) return;
    const int e = tile_entry(tf, cur, nxt, all, sc, l, t);
    if (e >= 0) tf.list[atomicAdd(tf.count, 1)] = e;
}

cudaError_t launch_tile_list(const TileFlags& tf, int cur, int nxt, int all, int skip0, int skip1,
                             const SubstepCount& sc, int* count_next, double* zero_ledger, unsigned int* zero_bits,
                             cudaStream_t st, const double* sum, double wet) {
    if (!count_next) {
        cudaError_t e = cudaMemsetAsync(tf.count, 0, sizeof(int), st);
        if (e != cudaSuccess) return e;
    }
    const int n = 2 * tf.tiles_x * tf.tiles_x;
    ::silt::launch_dep(k_tile_list, dim3((n + 255) / 256), dim3(256), 0, st, tf, cur, nxt, all, skip0, skip1, sc, count_next, zero_ledger,
                                                 zero_bits, sum, wet);
    ::silt::count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------- TMA staging of halo tiles

constexpr int TMA_WAIT_LIMIT = 1 << 22;  // mbarrier polls before a CTA gives up on a copy

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Waits for the barrier phase with a bounded number of polls; false if it
// never completed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done = 0;
    for (int k = 0; k < TMA_WAIT_LIMIT && !done; ++k)
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
    return done != 0;
}

// One 2D tile copy global -> this CTA's own shared memory only, counted
// on `bar`. x must be a multiple of 4 floats (16 bytes).
__device__ __forceinline__ void tma_load_2d(float* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_addr(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// The mbarrier of a CTA's tile copies and the parity of its next phase.
struct TileStage {
    uint64_t* bar;
    uint32_t phase;
    bool off;  // a copy did not arrive in time: this CTA loads its tiles itself
};

// h, u and v of a transport tile, rows [ty0-2, ty0+33) x columns
// [tx0-4, tx0+36), into their shared planes: three TMA copies (h, u, v
// tensor maps of the layer) completing one phase of the stage's barrier.
// Columns past the grid's edge read 0 and are not used. False when the copies
// did not arrive within the poll limit, twice: the error word gets bit 1 and
// the caller loads the planes itself.
__device__ bool tma_stage_transport(const CUtensorMap* maps, float* HSm, float* US, float* VS, int tx0, int ty0,
                                    TileStage& ts, unsigned int* err) {
    // Every thread's earlier writes of these planes come before the copies' writes.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(ts.bar)),
                     "r"(3 * TS * TW * (int)sizeof(float))
                     : "memory");
        tma_load_2d(HSm, maps + 0, tx0 - 4, ty0 - 2, ts.bar);
        tma_load_2d(US, maps + 1, tx0 - 4, ty0 - 2, ts.bar);
        tma_load_2d(VS, maps + 2, tx0 - 4, ty0 - 2, ts.bar);
    }
    bool ok = __syncthreads_and(mbar_wait(ts.bar, ts.phase) ? 1 : 0) != 0;
    if (!ok) ok = __syncthreads_and(mbar_wait(ts.bar, ts.phase) ? 1 : 0) != 0;
    if (!ok) {
        if (threadIdx.x == 0 && err) atomicOr(err, 2u);
        ts.off = true;  // the phases are no longer known: no more copies
        return false;
    }
    ts.phase ^= 1u;
    return true;
}

// Cells [x0, x1) x [y0, y1) of a transport tile, at most W x H of them, walked
// as one flat range of compile-time width so that every lane is busy on the
// 33-35 wide passes; interior tiles have exactly W x H, edge tiles fewer.
template <bool EDGE, int W, int H, class F>
__device__ __forceinline__ void trows(int x0, int x1, int y0, int y1, F f) {
    for (int k = threadIdx.x; k < W * H; k += TRANSPORT_THREADS) {
        const int r = k / W, gx = x0 + (k - r * W), gy = y0 + r;
        if (!EDGE || (gx < x1 && gy < y1)) f(gx, gy);
    }
}

// Donor-cell transport (src/fluid_core.rs:3025-3137), x pass then z pass on
// the updated depth, dry cut (src/fluid_core.rs:2072-2081), FP64 ledger sum.
// An edge moves depth one way only (the sign of its face speed picks the
// donor), so each flux pass evaluates the edges whose donor it is and writes
// 0 for the others. EDGE = false: the tile is full and its cells
// [t0-2, t1+1) lie inside the grid with t1 <= res-1, so no range is clipped.
template <bool EDGE>
__device__ __forceinline__ void transport_tile(const TransportParams& P, float* sm, int tx0, int ty0,
                                               const TileFlags& tf, int l, int nxt, int t, const CUtensorMap* maps,
                                               TileStage* ts) {
    const int res = P.res;
    const int tx1 = min(res, tx0 + TT), ty1 = min(res, ty0 + TT);
    constexpr int PL = TPL;
    float* HSm = sm;            // h on rows [ty0-2, ty1+1), cols [tx0-2, tx1+1)
    float* US = sm + PL;        // u on the same cells
    float* FL = sm + 2 * PL;    // left-going flux of edge e (cells e, e+1)
    float* FR = sm + 3 * PL;    // right-going flux
    float* HX = sm + 4 * PL;    // depth after the x pass
    float* VS = sm + 5 * PL;    // v
    float* UP = FL;             // up-going flux of row pair (r, r+1): the x fluxes are spent by then
    float* DN = FR;             // down-going flux
    const int ox = tx0 - 4, oy = ty0 - 2;
#define TIDX(gx, gy) (((gy) - oy) * TS + ((gx) - ox))
    const int ry0 = max(0, ty0 - 2), ry1 = min(res, ty1 + 1);
    const int cx0 = max(0, tx0 - 2), cx1 = min(res, tx1 + 1);
    const FixedDiv& cell = P.div_cell;
    const float dt = P.dt;
    const bool with_bed = P.bank_bed != nullptr;
    const uint8_t* gate = P.gate;
    // An interior tile of a layer with tensor maps arrives by TMA.
    const bool by_tma = !EDGE && maps && ts && !ts->off &&
                        tma_stage_transport(maps, HSm, US, VS, tx0, ty0, *ts, tf.sweep ? &tf.sweep->err : nullptr);
    if (!by_tma) {
        const float *h = P.h, *u = P.u, *v = P.v;
        trows<EDGE, TT + 3, TT + 3>(cx0, cx1, ry0, ry1, [&](int gx, int gy) {
            const size_t g = plane_index<size_t>(gx, gy, res);
            const int s = TIDX(gx, gy);
            stage(&HSm[s], h + g);
            stage(&US[s], u + g);
            if (gx >= tx0 && gx < tx1) stage(&VS[s], v + g);
        });
        staged();
        __syncthreads();
    }
    // x pass. Edge e joins cells e and e+1 and exists for 0 <= e < res-1.
    // Left-going flux first (its donor e+1 has removed nothing yet).
    const int e0 = max(0, tx0 - 2), e1 = min(res - 2, tx1 - 1);  // inclusive edge range
    trows<EDGE, TT + 2, TT + 3>(e0, e1 + 1, ry0, ry1, [&](int e, int gy) {
        float speed = 0.5f * (US[TIDX(e, gy)] + US[TIDX(e + 1, gy)]);
        float dh = 0.0f;
        if (!(speed > 0.0f)) {
            size_t g = (size_t)gy * res + e;
            float bd = with_bed ? P.bank_bed[g + 1] : 0.0f, bc = with_bed ? P.bank_bed[g] : 0.0f;
            dh = open_edge_dh(with_bed, HSm[TIDX(e + 1, gy)], HSm[TIDX(e, gy)], 0.0f, gate ? gate[g] : 1, bd, bc,
                              speed, dt, cell, 0.45f);
        }
        FL[TIDX(e, gy)] = dh;
    });
    __syncthreads();
    // Right-going: donor e has removed the left-going flux of edge e-1.
    trows<EDGE, TT + 1, TT + 3>(max(e0, tx0 - 1), e1 + 1, ry0, ry1, [&](int e, int gy) {
        float speed = 0.5f * (US[TIDX(e, gy)] + US[TIDX(e + 1, gy)]);
        float dh = 0.0f;
        if (speed > 0.0f) {
            float prev = e > 0 ? FL[TIDX(e - 1, gy)] : 0.0f;
            size_t g = (size_t)gy * res + e;
            float bd = with_bed ? P.bank_bed[g] : 0.0f, bc = with_bed ? P.bank_bed[g + 1] : 0.0f;
            dh = open_edge_dh(with_bed, HSm[TIDX(e, gy)], HSm[TIDX(e + 1, gy)], 0.0f + prev, gate ? gate[g + 1] : 1,
                              bd, bc, speed, dt, cell, 0.45f);
        }
        FR[TIDX(e, gy)] = dh;
    });
    __syncthreads();
    // Depth after the x pass on rows [ry0, ry1), tile columns. The rounding
    // book takes, for the tile's own cells, each cell's f32 change less the
    // exact (FP64) sum of the fluxes across its faces.
    double rnd = 0.0;
    const bool book_round = P.round != nullptr;
    trows<EDGE, TT, TT + 3>(tx0, tx1, ry0, ry1, [&](int c, int gy) {
        float flm = c - 1 >= 0 ? FL[TIDX(c - 1, gy)] : 0.0f;
        float frm = c - 1 >= 0 ? FR[TIDX(c - 1, gy)] : 0.0f;
        float flc = c <= res - 2 ? FL[TIDX(c, gy)] : 0.0f;
        float frc = c <= res - 2 ? FR[TIDX(c, gy)] : 0.0f;
        float rem = (0.0f + flm) + frc;
        float add = (0.0f + frm) + flc;
        float hv = HSm[TIDX(c, gy)];
        float moved = fmaxf(hv - rem + add, 0.0f);
        const float hx = (rem > 0.0f || add > 0.0f) ? moved : hv;
        HX[TIDX(c, gy)] = hx;
        if (book_round && gy >= ty0 && gy < ty1)
            rnd += ((double)hx - (double)hv) - (((double)frm + (double)flc) - ((double)flm + (double)frc));
    });
    __syncthreads();
    // z pass. Pair r joins rows r and r+1 and exists for 0 <= r < res-1.
    const int p0 = max(0, ty0 - 2), p1 = min(res - 2, ty1 - 1);
    trows<EDGE, TT, TT + 2>(tx0, tx1, p0, p1 + 1, [&](int c, int r) {
        float speed = 0.5f * (VS[TIDX(c, r)] + VS[TIDX(c, r + 1)]);
        float dh = 0.0f;
        if (!(speed > 0.0f)) {
            size_t g = (size_t)r * res + c;
            float bd = with_bed ? P.bank_bed[g + res] : 0.0f, bc = with_bed ? P.bank_bed[g] : 0.0f;
            dh = open_edge_dh(with_bed, HX[TIDX(c, r + 1)], HX[TIDX(c, r)], 0.0f, gate ? gate[g] : 1, bd, bc, speed,
                              dt, cell, 0.45f);
        }
        UP[TIDX(c, r)] = dh;
    });
    __syncthreads();
    trows<EDGE, TT, TT + 1>(tx0, tx1, max(p0, ty0 - 1), p1 + 1, [&](int c, int r) {
        float speed = 0.5f * (VS[TIDX(c, r)] + VS[TIDX(c, r + 1)]);
        float dh = 0.0f;
        if (speed > 0.0f) {
            float ra = r > 0 ? 0.0f + UP[TIDX(c, r - 1)] : 0.0f;
            size_t g = (size_t)r * res + c;
            float bd = with_bed ? P.bank_bed[g] : 0.0f, bc = with_bed ? P.bank_bed[g + res] : 0.0f;
            dh = open_edge_dh(with_bed, HX[TIDX(c, r)], HX[TIDX(c, r + 1)], ra, gate ? gate[g + res] : 1, bd, bc,
                              speed, dt, cell, 0.45f);
        }
        DN[TIDX(c, r)] = dh;
    });
    __syncthreads();
    double part = 0.0, cut = 0.0;
    trows<EDGE, TT, TT>(tx0, tx1, ty0, ty1, [&](int c, int r) {
        float upm = r - 1 >= 0 ? UP[TIDX(c, r - 1)] : 0.0f;
        float dnm = r - 1 >= 0 ? DN[TIDX(c, r - 1)] : 0.0f;
        float upc = r <= res - 2 ? UP[TIDX(c, r)] : 0.0f;
        float dnc = r <= res - 2 ? DN[TIDX(c, r)] : 0.0f;
        float rem = (0.0f + upm) + dnc;
        float add = (0.0f + dnm) + upc;
        float hv = HX[TIDX(c, r)];
        float moved = fmaxf(hv - rem + add, 0.0f);
        float hn = (rem > 0.0f || add > 0.0f) ? moved : hv;
        if (book_round)
            rnd += ((double)hn - (double)hv) - (((double)dnm + (double)upc) - ((double)upm + (double)dnc));
        if (P.eps > 0.0f && hn < P.eps) {
            if (hn > 0.0f) cut += (double)hn;  // booked: the dry cut's volume
            hn = 0.0f;
        }
        P.h_out[(size_t)r * res + c] = hn;
        part += (double)fmaxf(hn, 0.0f);
    });
    for (int o = 16; o > 0; o >>= 1) cut += __shfl_down_sync(0xffffffffu, cut, o);
    if ((threadIdx.x & 31) == 0 && cut > 0.0 && P.cut) atomicAdd(P.cut, cut * P.cut_area);
    if (book_round) {
        for (int o = 16; o > 0; o >>= 1) rnd += __shfl_down_sync(0xffffffffu, rnd, o);
        if ((threadIdx.x & 31) == 0 && rnd != 0.0) atomicAdd(P.round, rnd * P.cut_area);
    }
#undef TIDX
    // Block sum of the depth (FP64), one atomic per tile; the tile's flags.
    const int any = __syncthreads_or(part > 0.0);
    for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
    __shared__ double warp_sum[TRANSPORT_THREADS / 32];
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < (blockDim.x >> 5) ? warp_sum[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) {
            if (P.ledger) atomicAdd(P.ledger, v);
            pick(tf.wet, l, nxt)[t] = any ? 1 : 0;
            pick(tf.zero_h, l, nxt)[t] = any ? 0 : 1;
        }
    }
    __syncthreads();  // shared memory is reused by the next tile
}

// Identity substep of one depth tile: copy, ledger sum and flags as
// transport_tile leaves them.
__device__ void copy_tile(const TransportParams& P, int tx0, int ty0, const TileFlags& tf, int l, int nxt, int t) {
    const int res = P.res;
    const int w = min(TT, res - tx0), h = min(TT, res - ty0);
    double part = 0.0;
    for (int q = threadIdx.x; q < w * h; q += blockDim.x) {
        const size_t g = (size_t)(ty0 + q / w) * res + tx0 + q % w;
        const float hv = P.h[g];
        P.h_out[g] = hv;
        part += (double)fmaxf(hv, 0.0f);
    }
    const int any = __syncthreads_or(part > 0.0);
    for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
    __shared__ double warp_sum[TRANSPORT_THREADS / 32];
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < (blockDim.x >> 5) ? warp_sum[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) {
            if (P.ledger) atomicAdd(P.ledger, v);
            pick(tf.wet, l, nxt)[t] = any ? 1 : 0;
            pick(tf.zero_h, l, nxt)[t] = any ? 0 : 1;
        }
    }
    __syncthreads();
}

// One list entry of the transport pass.
__device__ __forceinline__ void transport_entry(const TransportParams& P, const TileFlags& tf, int nxt, int e,
                                                float* sm, const CUtensorMap* maps = nullptr,
                                                TileStage* ts = nullptr) {
    const int l = e >> 30, zero_fill = (e & ENTRY_ZERO) != 0, copy = (e & ENTRY_COPY) != 0, t = e & ENTRY_TILE;
    const int res = P.res;
    const int tx0 = (t % tf.tiles_x) * TT, ty0 = (t / tf.tiles_x) * TT;
    if (copy) {
        copy_tile(P, tx0, ty0, tf, l, nxt, t);
        return;
    }
    if (zero_fill) {
        const int w = min(TT, res - tx0), h = min(TT, res - ty0);
        for (int q = threadIdx.x; q < w * h; q += blockDim.x)
            P.h_out[(size_t)(ty0 + q / w) * res + tx0 + q % w] = 0.0f;
        if (threadIdx.x == 0) {
            pick(tf.wet, l, nxt)[t] = 0;
            pick(tf.zero_h, l, nxt)[t] = 1;
        }
        return;
    }
    const bool interior = tx0 >= 2 && ty0 >= 2 && tx0 + TT + 1 <= res && ty0 + TT + 1 <= res;
    if (interior)
        transport_tile<false>(P, sm, tx0, ty0, tf, l, nxt, t, maps, ts);
    else
        transport_tile<true>(P, sm, tx0, ty0, tf, l, nxt, t, nullptr, nullptr);
}

// Persistent over the substep's tile list.
__global__ void __launch_bounds__(TRANSPORT_THREADS, TRANSPORT_CTAS) k_transport(TransportLaunch L,
                                                                   const __grid_constant__ TransportMaps M) {
    ::silt::dep_wait();
    extern __shared__ __align__(128) float sm[];
    __shared__ TransportParams Ps[2];
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x < 2) {
        const int l = threadIdx.x;
        TransportParams P = L.lay[l];
        if (L.sc.speed2) P.dt = L.sc.dt / (float)device_nsub(L.sc, l);
        Ps[l] = P;
    }
    const bool tma = (M.on[0] || M.on[1]) && (smem_addr(sm) & 127u) == 0;
    if (tma && threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bar)), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    TileStage ts{&bar, 0u, !tma};
    const int n = *L.tf.count;
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const int e = L.tf.list[k];
        const int l = e >> 30;
        transport_entry(Ps[l], L.tf, L.nxt, e, sm, M.on[l] ? M.map[l] : nullptr, &ts);
    }
}

// Materialises the lazy dry cut: u = v = 0 where h < eps.
__global__ void k_apply_cut(const float* h, float* u, float* v, size_t n, float eps) {
    ::silt::dep_wait();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (h[i] < eps) { u[i] = 0.0f; v[i] = 0.0f; }
}

// Largest squared speed, for the CFL substep count (src/fluid_core.rs:1723-1744),
// and the depth sum of the wet test (:840-844), in one reading of the planes:
// as two passes they took 26 us of a flooded 1000^2 operator step's 214.
__global__ void __launch_bounds__(256) k_speed_sum(const float* h, const float* u, const float* v, size_t n,
                                                   unsigned int* bits, double* sum) {
    ::silt::dep_wait();
    float m = 0.0f;
    double s = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float uu = u[i], vv = v[i], hv = h[i];
        const float s2 = uu * uu + vv * vv;
        if (s2 > m) m = s2;
        s += (double)fmaxf(hv, 0.0f);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(bits, __float_as_uint(m));
    block_add(s, sum);
}

// One pass for what were three plane copies and the dry cut.
__global__ void __launch_bounds__(256) k_finish(const float* h1, const float* u1, const float* v1, float* h, float* u,
                                                float* v, size_t n, float eps, const double* sum, double wet) {
    ::silt::dep_wait();
    if (!(*sum > wet)) return;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float hv = h1[i], uu = u1[i], vv = v1[i];
        const bool dry = hv < eps;
        h[i] = hv;
        u[i] = dry ? 0.0f : uu;
        v[i] = dry ? 0.0f : vv;
    }
}

// The largest squared speed over the stepped tiles of substep 0's list (every tile that
// may hold water is one of them; a tile without water has no cell at or above
// eps and, after the dry cut, no velocity). Each thread loads its four cells
// before comparing, so a tile costs one memory round trip.
__global__ void __launch_bounds__(256) k_tile_speed2(TileFlags tf, const float* h0, const float* u0, const float* v0,
                                                     const float* h1, const float* u1, const float* v1, int res,
                                                     float eps, int apply_cut, unsigned int* bits) {
    ::silt::dep_wait();
    const int n = *tf.count;
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const int e = tf.list[k];
        if (e & (ENTRY_ZERO | ENTRY_COPY)) continue;
        const int l = e >> 30, t = e & ENTRY_TILE;
        const float* h = l ? h1 : h0;
        const float* u = l ? u1 : u0;
        const float* v = l ? v1 : v0;
        const int tx0 = (t % tf.tiles_x) * GRID_TILE, ty0 = (t / tf.tiles_x) * GRID_TILE;
        const int gx = tx0 + lane;
        float hv[4], uv[4], vv[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int gy = ty0 + wy + 8 * r;
            const bool in = gx < res && gy < res;
            const size_t g = in ? (size_t)gy * res + gx : 0;
            hv[r] = in ? h[g] : 0.0f;
            uv[r] = in ? u[g] : 0.0f;
            vv[r] = in ? v[g] : 0.0f;
        }
        float m = 0.0f;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (apply_cut && hv[r] < eps) continue;
            const float s2 = uv[r] * uv[r] + vv[r] * vv[r];
            if (s2 > m) m = s2;
        }
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
        if (lane == 0 && m > 0.0f) atomicMax(&bits[l], __float_as_uint(m));
    }
}

cudaError_t launch_tile_speed2(const TileFlags& tf, const float* const h[2], const float* const u[2],
                               const float* const v[2], int res, float eps, int apply_cut, unsigned int* bits,
                               cudaStream_t st) {
    ::silt::launch_dep(k_tile_speed2, dim3(148 * 8), dim3(256), 0, st, tf, h[0], u[0], v[0], h[1], u[1], v[1], res, eps, apply_cut, bits);
    ::silt::count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------ batched windows

__global__ void k_batch_tile_list(const WindowSubstep* ws, int* list, int* entry_win, int* count, int* count_next,
                                  SweepState* sweep) {
    ::silt::dep_wait();
    const int w = blockIdx.y;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (w == 0 && k == 0) {
        *count_next = 0;
        clear_sweep(sweep);
    }
    const WindowSubstep& D = ws[w];
    if (D.skip) return;
    const TileFlags& tf = D.F.tf;
    if (k == 0) {
        if (D.zero_ledger) D.zero_ledger[0] = D.zero_ledger[1] = 0.0;
        if (D.zero_bits) D.zero_bits[0] = D.zero_bits[1] = 0u;
    }
    const int nt = tf.tiles_x * tf.tiles_x;
    if (k >= 2 * nt) return;
    const int l = k / nt, t = k % nt;
    const int e = tile_entry(tf, D.cur, D.F.nxt, D.all, D.F.sc, l, t);
    if (e >= 0) {
        const int q = atomicAdd(count, 1);
        list[q] = e;
        entry_win[q] = w;
    }
}

__global__ void __launch_bounds__(256) k_batch_speed2(const WindowSubstep* ws, const int* list, const int* entry_win,
                                                      const int* count) {
    ::silt::dep_wait();
    const int n = *count;
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const int e = list[k];
        if (e & (ENTRY_ZERO | ENTRY_COPY)) continue;
        const WindowSubstep& D = ws[entry_win[k]];
        if (!D.zero_bits) continue;
        const int l = e >> 30, t = e & ENTRY_TILE;
        const LayerParams& P = D.F.lay[l];
        const int res = P.res, tiles_x = D.F.tf.tiles_x;
        const int tx0 = (t % tiles_x) * GRID_TILE, ty0 = (t / tiles_x) * GRID_TILE;
        const int gx = tx0 + lane;
        float hv[4], uv[4], vv[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int gy = ty0 + wy + 8 * r;
            const bool in = gx < res && gy < res;
            const size_t g = in ? (size_t)gy * res + gx : 0;
            hv[r] = in ? P.h[g] : 0.0f;
            uv[r] = in ? P.u[g] : 0.0f;
            vv[r] = in ? P.v[g] : 0.0f;
        }
        float m = 0.0f;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (D.apply_cut && hv[r] < P.eps) continue;
            const float s2 = uv[r] * uv[r] + vv[r] * vv[r];
            if (s2 > m) m = s2;
        }
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
        if (lane == 0 && m > 0.0f) atomicMax(&D.zero_bits[l], __float_as_uint(m));
    }
}

// (At three CTAs per SM its registers spill: two.)
__global__ void __launch_bounds__(FORCE_THREADS) k_batch_force(const WindowSubstep* ws, const int* list,
                                                               const int* entry_win, const int* count) {
    ::silt::dep_wait();
    extern __shared__ float sm[];
    __shared__ LayerParams Ps;
    __shared__ TileFlags Tf;
    __shared__ int nxt_s;
    const int n = *count;
    const WholeCta T;
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const int e = list[k];
        if (threadIdx.x == 0) {
            const WindowSubstep& D = ws[entry_win[k]];
            Ps = force_params(D.F.lay[e >> 30], D.F.sc, e >> 30, true);
            Tf = D.F.tf;
            nxt_s = D.F.nxt;
        }
        __syncthreads();
        if (!Ps.sweep) force_entry<Snap>(T, Ps, Tf, nxt_s, e, sm);  // the others are k_batch_force_sweep's
        __syncthreads();  // the parameters and shared memory are reused by the next entry
    }
}

// Every window's force pass in the sweep form, as force_sweep does for one
// sheet; a window in the snapshot form is k_batch_force's. Each team keeps
// its entry's parameters in its own slot.
struct BatchEntry {
    LayerParams P;
    TileFlags tf;
    int nxt;
};

template <class TM>
__device__ __forceinline__ void batch_force_sweep(const WindowSubstep* ws, int nwin, const int* list,
                                                  const int* entry_win, int n, SweepState* S, BatchEntry* slots,
                                                  float* sm) {
    const SweepTeam<TM> W(sm);
    BatchEntry& B = slots[W.half];
    auto fetch = [&](int k, bool report) {
        const int e = list[k];
        if (W.T.tid == 0) {
            const WindowSubstep& D = ws[entry_win[k]];
            B.P = force_params(D.F.lay[e >> 30], D.F.sc, e >> 30, report);
            B.tf = D.F.tf;
            B.nxt = D.F.nxt;
        }
        W.T.sync();
        return e;
    };
    for (int k = W.first; k < n; k += W.stride) {
        const int e = fetch(k, true);
        if (B.P.sweep) force_entry<Sweep>(W.T, B.P, B.tf, B.nxt, e, W.sm);
        W.T.sync();  // the parameters and shared memory are reused by the next entry
    }
    unsigned int target = 0;
    const unsigned int epoch = ld_acquire_u32(&S->epoch);
    if (!grid_barrier(S, target)) return;
    const bool reuse = n <= W.stride;  // one entry per team: its tile stays in shared memory
    const int passes = sweep_fixed_point(W, S, target, n, [&](int k, int pass) {
        const int e = fetch(k, false);
        const bool r = sweep_entry(W.T, B.P, B.tf, e, W.sm, pass, epoch, reuse);
        W.T.sync();
        return r;
    });
    if (passes < 0) return;
    if (passes == 0) {
        for (int u = blockIdx.x; u < 2 * nwin; u += gridDim.x) {
            if (threadIdx.x != 0) continue;
            const WindowSubstep& D = ws[u >> 1];
            const int l = u & 1;
            if (D.skip) continue;
            const LayerParams P = force_params(D.F.lay[l], D.F.sc, l, false);
            if (P.sweep && P.vort > 0.0f && !P.skip && layer_steps(D.F.sc, l)) sweep_serial(P);
        }
        if (!grid_barrier(S, target)) return;
    }
    sweep_stats(S, passes);
    for (int k = W.first; k < n; k += W.stride) {
        const int e = fetch(k, false);
        post_entry(W.T, B.P, B.tf, e, W.sm);
        W.T.sync();
    }
}

__global__ void __launch_bounds__(FORCE_THREADS, 2) k_batch_force_sweep(const WindowSubstep* ws, int nwin,
                                                                        const int* list, const int* entry_win,
                                                                        const int* count, SweepState* S) {
    ::silt::dep_wait();
    extern __shared__ float sm[];
    __shared__ BatchEntry slots[2];
    const int n = *count;
    if (n <= (int)gridDim.x)
        batch_force_sweep<WholeCta>(ws, nwin, list, entry_win, n, S, slots, sm);
    else
        batch_force_sweep<HalfCta>(ws, nwin, list, entry_win, n, S, slots, sm);
}

__global__ void __launch_bounds__(TRANSPORT_THREADS, TRANSPORT_CTAS) k_batch_transport(const WindowSubstep* ws, const int* list,
                                                                       const int* entry_win, const int* count) {
    ::silt::dep_wait();
    extern __shared__ float sm[];
    __shared__ TransportParams Ps;
    __shared__ TileFlags Tf;
    __shared__ int nxt_s;
    const int n = *count;
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const int e = list[k];
        if (threadIdx.x == 0) {
            const WindowSubstep& D = ws[entry_win[k]];
            const int l = e >> 30;
            TransportParams P = D.T.lay[l];
            if (D.T.sc.speed2) P.dt = D.T.sc.dt / (float)device_nsub(D.T.sc, l);
            Ps = P;
            Tf = D.T.tf;
            nxt_s = D.T.nxt;
        }
        __syncthreads();
        transport_entry(Ps, Tf, nxt_s, e, sm);
        __syncthreads();
    }
}

cudaError_t launch_batch_tile_list(const WindowSubstep* d_ws, int nwin, int max_tiles, int* list, int* entry_win,
                                   int* count, int* count_next, SweepState* sweep, cudaStream_t st) {
    if (nwin <= 0) return cudaSuccess;
    dim3 grid((2 * max_tiles + 255) / 256, nwin);
    ::silt::launch_dep(k_batch_tile_list, dim3(grid), dim3(256), 0, st, d_ws, list, entry_win, count, count_next,
                       sweep);
    ::silt::count_launch();
    return cudaGetLastError();
}

cudaError_t launch_batch_speed2(const WindowSubstep* d_ws, const int* list, const int* entry_win, const int* count,
                                cudaStream_t st) {
    ::silt::launch_dep(k_batch_speed2, dim3(148 * 8), dim3(256), 0, st, d_ws, list, entry_win, count);
    ::silt::count_launch();
    return cudaGetLastError();
}

// CTAs of a cooperative force launch that the current device holds at once;
// not positive when it cannot be told (the launch is refused then).
template <class... KArgs>
int coop_grid(void (*kernel)(KArgs...), int dev) {
    int per = 0;
    if (allow_smem(kernel, SWEEP_SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, FORCE_THREADS, SWEEP_SMEM) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return query_sm_count(dev) * per;
}

template <class K, class... Args>
cudaError_t launch_coop(K kernel, int grid, cudaStream_t st, Args... args) {
    if (grid <= 0) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(FORCE_THREADS);
    cfg.dynamicSmemBytes = SWEEP_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = ::silt::launch_ex(cfg, kernel, args...);
    ::silt::count_launch();
    return e;
}

cudaError_t launch_batch_force(const WindowSubstep* d_ws, int nwin, const int* list, const int* entry_win,
                               const int* count, SweepState* sweep, bool snapshot, cudaStream_t st, int ctas_per_sm) {
    if (sweep) {
        static PerDevice<int> grids, sms;
        const int dev = current_device();
        const int grid = grids.of(dev, [](int d) { return coop_grid(k_batch_force_sweep, d); });
        const int nsm = sms.of(dev, query_sm_count);
        // Fewer CTAs than the device holds stay co-resident: the launch is still cooperative.
        const int g = ctas_per_sm > 0 ? std::min(grid, ctas_per_sm * nsm) : grid;
        const cudaError_t e = launch_coop(k_batch_force_sweep, g, st, d_ws, nwin, list, entry_win, count, sweep);
        if (e != cudaSuccess || !snapshot) return e != cudaSuccess ? e : cudaGetLastError();
    }
    static PerDevice<cudaError_t> attr;
    const cudaError_t allowed = attr.of(current_device(), [](int) { return allow_smem(k_batch_force, Snap::BYTES); });
    if (allowed != cudaSuccess) return allowed;
    ::silt::launch_dep(k_batch_force, dim3(148 * 2), dim3(FORCE_THREADS), Snap::BYTES, st, d_ws, list, entry_win, count);
    ::silt::count_launch();
    return cudaGetLastError();
}

cudaError_t launch_batch_transport(const WindowSubstep* d_ws, const int* list, const int* entry_win,
                                   const int* count, cudaStream_t st, int blocks) {
    static PerDevice<cudaError_t> attr;
    const cudaError_t allowed = attr.of(current_device(), [](int) { return allow_smem(k_batch_transport, transport_smem_bytes()); });
    if (allowed != cudaSuccess) return allowed;
    const unsigned grid = blocks > 0 ? (unsigned)blocks : 148u * 4u;
    ::silt::launch_dep(k_batch_transport, dim3(grid), dim3(TRANSPORT_THREADS), transport_smem_bytes(), st, d_ws, list, entry_win, count);
    ::silt::count_launch();
    return cudaGetLastError();
}

cudaError_t launch_force(const ForceLaunch& L, int res, int layers, cudaStream_t st) {
    if (L.lay[0].sweep || L.lay[1].sweep) {
        if (!L.tf.sweep) return cudaErrorInvalidValue;
        static PerDevice<int> grids;
        const int grid = grids.of(current_device(), [](int d) { return coop_grid(k_force_sweep, d); });
        const cudaError_t e = launch_coop(k_force_sweep, grid, st, L);
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    (void)layers;
    static_assert(FarSnap::BYTES == Snap::BYTES, "one tile layout");
    static PerDevice<cudaError_t> attr;
    const cudaError_t allowed = attr.of(current_device(), [](int) {
        const cudaError_t e = allow_smem(k_force, Snap::BYTES);
        return e != cudaSuccess ? e : allow_smem(k_force_far, Snap::BYTES);
    });
    if (allowed != cudaSuccess) return allowed;
    ::silt::launch_dep(res > MAX_NEAR_RES ? k_force_far : k_force, dim3(148 * SNAP_CTAS), dim3(FORCE_THREADS),
                       Snap::BYTES, st, L);
    ::silt::count_launch();
    return cudaGetLastError();
}

namespace {

// cuTensorMapEncodeTiled from the driver (through the runtime: no link to libcuda).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

// The transport's tensor map of a res x res FP32 plane: boxes of TS x TW
// cells, out-of-grid cells read as 0. Maps are kept per (plane, res): the
// step alternates between a few fixed buffers.
bool transport_map(const float* plane, int res, CUtensorMap* out) {
    struct Entry {
        const float* plane;
        int res;
        CUtensorMap map;
    };
    static std::mutex m;
    static std::vector<Entry> cache;
    std::lock_guard<std::mutex> lock(m);
    for (const Entry& e : cache)
        if (e.plane == plane && e.res == res) {
            *out = e.map;
            return true;
        }
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc || (res % 4) != 0 || (reinterpret_cast<uintptr_t>(plane) % 16) != 0) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)res, (cuuint64_t)res};
    const cuuint64_t strides[1] = {(cuuint64_t)res * sizeof(float)};
    const cuuint32_t box[2] = {(cuuint32_t)TS, (cuuint32_t)TW};
    const cuuint32_t elem[2] = {1, 1};
    Entry e{plane, res, {}};
    if (enc(&e.map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(plane), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    if (cache.size() >= 64) cache.erase(cache.begin());
    cache.push_back(e);
    *out = e.map;
    return true;
}

}  // namespace

cudaError_t launch_transport(const TransportLaunch& L, int res, int layers, cudaStream_t st) {
    static PerDevice<cudaError_t> attr;
    const cudaError_t allowed = attr.of(current_device(), [](int) { return allow_smem(k_transport, transport_smem_bytes()); });
    if (allowed != cudaSuccess) return allowed;
    (void)layers;
    // Interior tiles of a grid a multiple of 4 cells wide arrive by TMA.
    TransportMaps M;
    for (int l = 0; l < 2; ++l) {
        const TransportParams& P = L.lay[l];
        M.on[l] = P.res == res && P.h && P.u && P.v && transport_map(P.h, res, &M.map[l][0]) &&
                  transport_map(P.u, res, &M.map[l][1]) && transport_map(P.v, res, &M.map[l][2]);
    }
    ::silt::launch_dep(k_transport, dim3(148 * TRANSPORT_CTAS), dim3(TRANSPORT_THREADS), transport_smem_bytes(), st, L, M);
    ::silt::count_launch();
    return cudaGetLastError();
}

__global__ void k_material(const uint8_t* grain, const float* moisture, float* nu, float* mob, float* damp, size_t n) {
    ::silt::dep_wait();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float x = dynamic_viscosity(grain[i], moisture[i]);
        nu[i] = x;
        mob[i] = sheet_mobility_for(x);
        damp[i] = sheet_damp(x);
    }
}

cudaError_t launch_material(const uint8_t* grain, const float* moisture, float* nu, float* mob, float* damp, size_t n,
                            cudaStream_t st) {
    int blocks = (int)((n + 255) / 256);
    if (blocks > 148 * 16) blocks = 148 * 16;
    ::silt::launch_dep(k_material, dim3(blocks), dim3(256), 0, st, grain, moisture, nu, mob, damp, n);
    ::silt::count_launch();
    return cudaGetLastError();
}

cudaError_t launch_apply_cut(const float* h, float* u, float* v, size_t n, float eps, cudaStream_t st) {
    int blocks = (int)((n + 255) / 256);
    if (blocks > 148 * 16) blocks = 148 * 16;
    ::silt::launch_dep(k_apply_cut, dim3(blocks), dim3(256), 0, st, h, u, v, n, eps);
    ::silt::count_launch();
    return cudaGetLastError();
}

cudaError_t launch_speed_sum(const float* h, const float* u, const float* v, size_t n, unsigned int* bits, double* sum,
                             cudaStream_t st) {
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 8);
    ::silt::launch_dep(k_speed_sum, dim3(blocks), dim3(256), 0, st, h, u, v, n, bits, sum);
    ::silt::count_launch();
    return cudaGetLastError();
}

cudaError_t launch_finish(const float* h1, const float* u1, const float* v1, float* h, float* u, float* v, size_t n,
                          float eps, const double* sum, double wet, cudaStream_t st) {
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
    ::silt::launch_dep(k_finish, dim3(blocks), dim3(256), 0, st, h1, u1, v1, h, u, v, n, eps, sum, wet);
    ::silt::count_launch();
    return cudaGetLastError();
}

}  // namespace silt
