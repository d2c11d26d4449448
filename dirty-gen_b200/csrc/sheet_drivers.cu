// The coarse window's boundary drivers of open water: the paddle strip
// (src/fluid_core.rs:7420-7480 drive_waves) and the river reach's inlet and
// outlet (:7638-7745 feed_reach).
#include "sheet_drivers.cuh"

#include "block_sum.cuh"
#include "launch_count.cuh"

namespace silt {
namespace drivers {

namespace {

// Every water cell of the strip relaxes toward the paddle stroke along the
// push direction, the pull tapered over the strip's outer quarters; cells
// under 2 cm of water are left alone (so the lazy dry cut never matters).
__global__ void k_wave(fine::SheetView W, WaveStep w) {
    ::silt::dep_wait();
    const int ni = w.i1 - w.i0, nj = w.j1 - w.j0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < ni * nj; q += gridDim.x * blockDim.x) {
        const int i = w.i0 + q % ni, j = w.j0 + q / ni;
        const float x = W.origin[0] + ((float)i + 0.5f) * W.cell;
        const float z = W.origin[1] + ((float)j + 0.5f) * W.cell;
        if (x < w.x0 || x > w.x1 || z < w.z0 || z > w.z1) continue;
        const size_t idx = (size_t)j * W.res + i;
        const float h = W.h[0][idx];
        if (h < 0.02f || !isfinite(h)) continue;
        const float tx = fminf(fmaxf(fminf(x - w.x0, w.x1 - x) / (0.25f * w.span_x), 0.0f), 1.0f);
        const float tz = fminf(fmaxf(fminf(z - w.z0, w.z1 - z) / (0.25f * w.span_z), 0.0f), 1.0f);
        const float k = w.pull * fminf(tx, tz);
        const float u = W.u[0][idx], v = W.v[0][idx];
        const float along = u * w.dx + v * w.dz;
        const float d = (w.stroke - along) * k;
        const float nu = u + d * w.dx, nv = v + d * w.dz;
        if (isfinite(nu) && isfinite(nv)) {
            W.u[0][idx] = nu;
            W.v[0][idx] = nv;
        }
    }
}

// feed_reach (src/fluid_core.rs:7638-7757): the outlet's cells (cross-major),
// then the inlet's (row-major), each drawn toward its stage through the f32
// bank. The reference's sweep is sequential, since a cell reads the bank the
// one before left; but only the bank is. One block takes the cells in chunks:
// all threads read them, one thread walks the bank over the staged depths in
// the reference's order, all threads write. A cell then
// costs the walk some 50 cycles instead of a chain of global reads: the 320
// cells of a 4-row reach 8 m wide took 131 us, now 22.
constexpr int REACH_THREADS = 256, REACH_PER = 4, REACH_CHUNK = REACH_THREADS * REACH_PER;

__global__ void __launch_bounds__(REACH_THREADS) k_reach(fine::SheetView W, ReachStep r, float* bank, double* books) {
    ::silt::dep_wait();
    static_assert(REACH_CHUNK % 8 == 0, "the walk reads eight cells at a time");
    __shared__ float s_h[REACH_CHUNK];      // depth
    __shared__ float s_t[REACH_CHUNK];      // the stage's depth, -1 for a cell left alone
    __shared__ float s_new[REACH_CHUNK];    // depth after
    __shared__ unsigned int s_deep;
    const int tid = threadIdx.x, res = W.res;
    const float area = W.cell * W.cell, per_area = 1.0f / area;
    auto at = [&](int along, int cross) -> size_t {
        return r.along_z ? (size_t)along * res + cross : (size_t)cross * res + along;
    };
    auto row = [&](int k) { return r.positive ? k : res - 1 - k; };
    const int width = r.c1 - r.c0, first_out = res - r.rows;
    const long long half = (long long)width * r.rows;
    // The deepest inlet cell.
    if (tid == 0) s_deep = 0u;
    __syncthreads();
    float deepest = 0.0f;
    for (int c = r.c0 + tid; c < r.c1; c += REACH_THREADS)
        deepest = fmaxf(deepest, fmaxf(r.inlet_eta - W.bed[at(row(0), c)], 0.0f));
    atomicMax(&s_deep, __float_as_uint(deepest));  // non-negative floats order as their bits
    __syncthreads();
    const float deep = __uint_as_float(s_deep);
    const long long cells = deep > 0.0f ? 2 * half : half;
    float b = *bank;
    double moved = 0.0, inflow_m3 = 0.0;
    for (long long base = 0; base < cells; base += REACH_CHUNK) {
        const int n = (int)min((long long)REACH_CHUNK, cells - base);
        size_t idx[REACH_PER];
        float su[REACH_PER], sv[REACH_PER];
#pragma unroll
        for (int e = 0; e < REACH_PER; ++e) {
            const int q = tid + e * REACH_THREADS;
            const long long k = base + q;
            su[e] = sv[e] = 0.0f;
            idx[e] = 0;
            if (q >= n) continue;
            const bool out = k < half;
            float eta;
            if (out) {
                const int cross = r.c0 + (int)(k / r.rows);
                idx[e] = at(row(first_out + (int)(k % r.rows)), cross);
                const size_t src = at(row(first_out - 1), cross);
                su[e] = W.u[0][src];
                sv[e] = W.v[0][src];
                if (W.cut_pending && W.h[0][src] < 1.0e-6f) su[e] = sv[e] = 0.0f;  // the lazy dry cut of the copied cell
                eta = r.outlet_eta;
            } else {
                const long long m = k - half;
                idx[e] = at(row((int)(m / width)), r.c0 + (int)(m % width));
                eta = r.inlet_eta;
            }
            const float target = fmaxf(eta - W.bed[idx[e]], 0.0f), h = W.h[0][idx[e]];
            s_h[q] = h;
            s_t[q] = isfinite(h) && target > 0.0f ? target : -1.0f;
        }
        __syncthreads();
        if (tid == 0) {
            // Eight cells' depths at a time, so that only the bank's own chain
            // stands between one cell and the next.
            for (int q0 = 0; q0 < n; q0 += 8) {
                float h[8], t[8], h1[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    h[e] = s_h[q0 + e];
                    t[e] = q0 + e < n ? s_t[q0 + e] : -1.0f;
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    h1[e] = h[e];
                    if (!(t[e] >= 0.0f)) continue;
                    if (h[e] > t[e]) {
                        b += (h[e] - t[e]) * area;
                        h1[e] = t[e];
                    } else if (b > 0.0f) {
                        // min(need, b / area), without the division while the bank holds plainly more.
                        const float need = t[e] - h[e];
                        const float add = need < 0.999f * (b * per_area) ? need : fminf(need, b / area);
                        h1[e] = h[e] + add;
                        b -= add * area;
                    }
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) s_new[q0 + e] = h1[e];
            }
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < REACH_PER; ++e) {
            const int q = tid + e * REACH_THREADS;
            if (q >= n) continue;
            if (!(s_t[q] >= 0.0f)) continue;
            const size_t g = idx[e];
            const int i = (int)(g % res), j = (int)(g / res);
            const float h1 = s_new[q];
            if (h1 != s_h[q]) {
                W.h[0][g] = h1;
                moved += (double)h1 - (double)s_h[q];
                fine::mark_tile(W, 0, i, j);
            }
            if (base + q < half) {
                if (isfinite(su[e]) && isfinite(sv[e])) {
                    const float along = fmaxf(su[e] * r.dx + sv[e] * r.dz, 0.0f);
                    const float cross_v = r.along_z ? su[e] : sv[e];
                    W.u[0][g] = r.along_z ? cross_v : along * r.dx;
                    W.v[0][g] = r.along_z ? along * r.dz : cross_v;
                    fine::mark_tile(W, 0, i, j);
                }
            } else {
                const float speed = r.inlet_speed * sqrtf(fminf(fmaxf(h1 / deep, 0.0f), 1.0f));
                W.u[0][g] = speed * r.dx;
                W.v[0][g] = speed * r.dz;
                fine::mark_tile(W, 0, i, j);
                if (r.inflow_c > 0.0f) {
                    // The water arrives carrying its load (src/fluid_core.rs:7746-7755).
                    const float want = r.inflow_c * h1;
                    const float have = r.susp[g];
                    if (h1 >= 1.0e-5f && isfinite(have) && have < want) {
                        r.susp[g] = want;
                        inflow_m3 += (double)((want - have) * area);
                    }
                }
            }
        }
        __syncthreads();  // the staged cells are rewritten by the next chunk
    }
    // FP64 sums over the block: a serial chain of FP64 adds costs more than the walk.
    moved = block_sum(moved);
    inflow_m3 = block_sum(inflow_m3);
    if (tid != 0) return;
    if (inflow_m3 != 0.0) *r.entrained += inflow_m3;
    *bank = b;
    if (moved != 0.0) {
        if (W.d_acc) W.d_acc[0] += moved;
        books[4] -= moved * ((double)W.cell * (double)W.cell);
    }
}

}  // namespace

cudaError_t wave_step(const fine::SheetView& W, const WaveStep& w, cudaStream_t st) {
    const int n = (w.i1 - w.i0) * (w.j1 - w.j0);
    if (n <= 0) return cudaSuccess;
    const int blocks = (n + 255) / 256 < 296 ? (n + 255) / 256 : 296;
    ::silt::launch_dep(k_wave, dim3(blocks), dim3(256), 0, st, W, w);
    ::silt::count_launch();
    return cudaGetLastError();
}

cudaError_t reach_step(const fine::SheetView& W, const ReachStep& r, float* bank, double* books, cudaStream_t st) {
    if (r.c1 <= r.c0) return cudaSuccess;
    ::silt::launch_dep(k_reach, dim3(1), dim3(REACH_THREADS), 0, st, W, r, bank, books);
    ::silt::count_launch();
    return cudaGetLastError();
}

}  // namespace drivers
}  // namespace silt
