// Quadric surface grid: separable layers -> 7-coefficient cells (forward/backward) and the
// SDF / normal samples of a cell (kernel/surface.cu).
//
// Cell layout [R^3][7] fp32, index x + yR + zR^2; coefficients a0..a6 of
// f(u) = a0 ux^2 + a1 uy^2 + a2 uz^2 + a3 ux + a4 uy + a5 uz + a6 in local u in [-1,1)^3.
#include "common.cuh"

namespace qsdvr {

QSDVR_ERROR_WORD_ACCESSOR(surface)

namespace {

// ---- LayerToGrid ------------------------------------------------------------------------

// kernel/surface.cu:161-178: the per-axis prefix recurrences, evaluated with the same unfused
// float operations as the reference's host code:
//   a3[i] = (2 a0[i-1] + 2 a0[i]) + a3[i-1],
//   a6[i] = ((3 a0[i-1] + a0[i]) + 2 a3[i-1]) + a6[i-1].
// One block, one warp per axis.  The recurrences are bound by their serial chain, so only the
// chain is serial: a layer is staged in shared memory and the terms that need no earlier result
// (the parenthesised sums over a0) are formed by the whole warp, then one lane adds them up, one
// add per step and chain, from shared memory.  With the layer read and the results written in
// global memory inside the chain, each step waited for both (13.6 us at R = 256 for the separable tables, 8.0 us now; the chain's
// own adds are about 4 of them).
constexpr int kAxisThreads = 3 * kWarp;
inline size_t axis_smem(uint32_t R, int arrays) { return (size_t)3 * arrays * R * sizeof(float); }

// s3, s6 [R] of one axis in shared memory: on return a3 and a6.
__device__ __forceinline__ void axis_recurrence(const float *__restrict__ a0, float offset, uint32_t R, int lane,
                                                float *s3, float *s6) {
    for (uint32_t i = lane; i < R; i += kWarp) {
        const float c = a0[i], b = i ? a0[i - 1] : 0.0f;
        s3[i] = i ? __fadd_rn(__fmul_rn(2.0f, b), __fmul_rn(2.0f, c)) : offset;
        s6[i] = i ? __fadd_rn(__fmul_rn(3.0f, b), c) : 0.0f;
    }
    __syncwarp();
    if (lane == 0) {
        float p3 = s3[0], p6 = s6[0];
#pragma unroll 8
        for (uint32_t i = 1; i < R; ++i) {
            const float t6 = __fadd_rn(s6[i], __fmul_rn(2.0f, p3));
            p3 = __fadd_rn(s3[i], p3);
            p6 = __fadd_rn(t6, p6);
            s3[i] = p3;
            s6[i] = p6;
        }
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kAxisThreads) layer_tables_kernel(const float *__restrict__ x0,
                                                                    const float *__restrict__ y1,
                                                                    const float *__restrict__ z2,
                                                                    const float *__restrict__ offset, uint32_t R,
                                                                    float *__restrict__ tables
                                                                    /* [6][R]: x3 y4 z5 x6 y6 z6 */) {
    extern __shared__ float axis_s[];
    const int axis = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const float *a0 = axis == 0 ? x0 : (axis == 1 ? y1 : z2);
    float *s3 = axis_s + (size_t)2 * axis * R, *s6 = s3 + R;
    axis_recurrence(a0, offset[axis], R, lane, s3, s6);
    for (uint32_t i = lane; i < R; i += kWarp) {
        tables[axis * R + i] = s3[i];
        tables[(3 + axis) * R + i] = s6[i];
    }
}

// kernel/surface.cu:3-24: a block writes whole rows (7 R consecutive floats of one (y, z)), a
// thread one float at a time, so the stores coalesce.  The x terms (comps 0, 3, 6) come from
// shared memory, the row's own (1, 2, 4, 5) are seven floats there, and the choice is two
// selects: no 64-bit divisions to find the cell and no branch per component, which bound the
// kernel before (123 us at R = 128 for 59 MB of output; 28 us now).
__global__ void __launch_bounds__(256) layer_expand_kernel(float *__restrict__ grid7, const float *__restrict__ x0,
                                                           const float *__restrict__ y1,
                                                           const float *__restrict__ z2,
                                                           const float *__restrict__ tables,
                                                           const float *__restrict__ offset, uint32_t R) {
    extern __shared__ float xs[];  // [3][R]: x0, x3, x6
    __shared__ float rowc[2][7];   // the row's constants, the next row's written while this one is
    const float off3 = offset[3];
    const uint32_t n = 7 * R, t = threadIdx.x;
    for (uint32_t x = t; x < R; x += 256) {
        xs[x] = x0[x];
        xs[R + x] = tables[x];
        xs[2 * R + x] = tables[3 * R + x];
    }
    int buf = 0;
    for (uint32_t row = blockIdx.x; row < R * R; row += gridDim.x, buf ^= 1) {
        const uint32_t y = row % R, z = row / R;
        if (t < 7) {
            const float *src = t == 1 ? y1 + y
                                      : (t == 2 ? z2 + z : (t == 4 ? tables + R + y : tables + 2 * R + z));
            rowc[buf][t] = *src;
        }
        const float y6 = tables[4 * R + y], z6 = tables[5 * R + z];
        __syncthreads();
        float *out = grid7 + (uint64_t)row * n;
        for (uint32_t i = t; i < n; i += 256) {
            const uint32_t x = i / 7, comp = i - 7 * x, k = comp / 3;
            const float v = xs[k * R + x], w = rowc[buf][comp];
            const float sum = __fadd_rn(__fadd_rn(__fadd_rn(v, y6), z6), off3);
            out[i] = comp == 6 ? sum : (comp == 3 * k ? v : w);
        }
    }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// kernel/surface.cu:26-52 as a reduction.  A block takes a run of consecutive (z, y) rows, a
// thread one x (and every 256th after it): per-x sums over the rows stay in registers, per-y
// sums over x are warp-reduced and added up in shared memory, per-z sums stay in registers until
// z changes.  A row is summed over x 256 columns at a time, so a grid of any R keeps every warp
// busy, and the number of runs (kReduceBlocks, 8 resident blocks for each of 148 SMs) sets the
// number of global atomics instead of R: one block per z slab left most of the chip idle and
// half of each block's warps at R = 128 (98 us for 59 MB; 18 us now).
// acc layout: [0..3R) x3 y4 z5, [3R..6R) x6 y6 z6.
constexpr uint32_t kReduceBlocks = 148 * 8;

__global__ void __launch_bounds__(256) layer_grad_reduce_kernel(const float *__restrict__ g7, uint32_t R,
                                                                uint32_t rows_per_block, float *__restrict__ xg,
                                                                float *__restrict__ yg, float *__restrict__ zg,
                                                                float *__restrict__ acc, float *__restrict__ off3) {
    extern __shared__ float ysum[];  // [rows_per_block][3]: comps 1, 4, 6 summed over x
    const uint32_t first = blockIdx.x * rows_per_block;
    const uint32_t last = min(first + rows_per_block, R * R);
    if (first >= last) return;
    const int lane = threadIdx.x & 31;
    for (uint32_t i = threadIdx.x; i < 3 * rows_per_block; i += blockDim.x) ysum[i] = 0.0f;
    __syncthreads();
    for (uint32_t xb = 0; xb < R; xb += blockDim.x) {
        const uint32_t x = xb + threadIdx.x;
        const bool on = x < R;
        if (x - lane >= R) break;  // the whole warp is past the row
        float s0 = 0.0f, s3 = 0.0f, s6 = 0.0f;
        float z2 = 0.0f, z5 = 0.0f, z6 = 0.0f;
        uint32_t z = first / R;
        uint32_t left = (z + 1) * R - first;  // rows up to the next z
        for (uint32_t row = first; row < last; row += 4) {  // the loads of four rows in flight
            float v[4][7];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool have = on && row + u < last;
                const float *c = g7 + ((uint64_t)(row + u) * R + x) * 7;
#pragma unroll
                for (int k = 0; k < 7; ++k) v[u][k] = have ? c[k] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (row + u >= last) break;
                s0 += v[u][0];
                s3 += v[u][3];
                s6 += v[u][6];
                z2 += v[u][2];
                z5 += v[u][5];
                z6 += v[u][6];
                const float w1 = warp_sum(v[u][1]), w4 = warp_sum(v[u][4]), w6 = warp_sum(v[u][6]);
                if (lane < 3)
                    atomicAdd(&ysum[3 * (row + u - first) + lane], lane == 0 ? w1 : (lane == 1 ? w4 : w6));
                if (--left == 0 || row + u + 1 == last) {
                    const float t2 = warp_sum(z2), t5 = warp_sum(z5), t6 = warp_sum(z6);
                    if (lane < 4) {
                        float *p = lane == 0 ? zg + z
                                             : (lane == 1 ? acc + 2 * R + z : (lane == 2 ? acc + 5 * R + z : off3));
                        atomicAdd(p, lane == 0 ? t2 : (lane == 1 ? t5 : t6));
                    }
                    z2 = z5 = z6 = 0.0f;
                    ++z;
                    left = R;
                }
            }
        }
        if (on) {
            atomicAdd(&xg[x], s0);
            atomicAdd(&acc[x], s3);          // x3
            atomicAdd(&acc[3 * R + x], s6);  // x6
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < last - first; i += blockDim.x) {
        const uint32_t y = (first + i) % R;
        atomicAdd(&yg[y], ysum[3 * i]);
        atomicAdd(&acc[R + y], ysum[3 * i + 1]);      // y4
        atomicAdd(&acc[4 * R + y], ysum[3 * i + 2]);  // y6
    }
}

// kernel/surface.cu:301-334, the reverse recurrences of one axis, unfused as on the host, on its
// sums g0, g3, g6 [R] in shared memory.  In the reference's order, for i = R-1 down to 1:
//   g0[i] += g6[i]; g0[i-1] += 3 g6[i]; g3[i-1] += 2 g6[i]; g6[i-1] += g6[i],
// then the same with g0[i] += 2 g3[i]; g0[i-1] += 2 g3[i]; g3[i-1] += g3[i].  Only g6's and then
// g3's suffix sums are serial (one lane); each g0[i] then takes its terms in that order, all i
// at once: first the one from i + 1, then its own.
__device__ __forceinline__ void axis_reverse(float *g0, float *g3, float *g6, uint32_t R, int lane) {
    __syncwarp();
    if (lane == 0) {
        float c = g6[R - 1];
#pragma unroll 8
        for (uint32_t i = R - 1; i > 0; --i) {
            c = __fadd_rn(g6[i - 1], c);
            g6[i - 1] = c;
        }
    }
    __syncwarp();
    for (uint32_t i = lane; i < R; i += kWarp) {
        float v = g0[i];
        if (i + 1 < R) {
            v = __fadd_rn(v, __fmul_rn(3.0f, g6[i + 1]));
            g3[i] = __fadd_rn(g3[i], __fmul_rn(2.0f, g6[i + 1]));
        }
        if (i > 0) v = __fadd_rn(v, g6[i]);
        g0[i] = v;
    }
    __syncwarp();
    if (lane == 0) {
        float c = g3[R - 1];
#pragma unroll 8
        for (uint32_t i = R - 1; i > 0; --i) {
            c = __fadd_rn(g3[i - 1], c);
            g3[i - 1] = c;
        }
    }
    __syncwarp();
    for (uint32_t i = lane; i < R; i += kWarp) {
        float v = g0[i];
        if (i + 1 < R) v = __fadd_rn(v, __fmul_rn(2.0f, g3[i + 1]));
        if (i > 0) v = __fadd_rn(v, __fmul_rn(2.0f, g3[i]));
        g0[i] = v;
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kAxisThreads) layer_grad_reverse_kernel(float *__restrict__ xg,
                                                                          float *__restrict__ yg,
                                                                          float *__restrict__ zg,
                                                                          const float *__restrict__ acc,
                                                                          float *__restrict__ offset_grad, uint32_t R) {
    extern __shared__ float axis_s[];
    const int axis = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    float *a0 = axis == 0 ? xg : (axis == 1 ? yg : zg);
    float *g0 = axis_s + (size_t)3 * axis * R, *g3 = g0 + R, *g6 = g3 + R;
    for (uint32_t i = lane; i < R; i += kWarp) {
        g0[i] = a0[i];
        g3[i] = acc[axis * R + i];
        g6[i] = acc[(3 + axis) * R + i];
    }
    axis_reverse(g0, g3, g6, R, lane);
    for (uint32_t i = lane; i < R; i += kWarp) a0[i] = g0[i];
    if (lane == 0) offset_grad[axis] = g3[0];
}

// ---- separable SDF tables for the fused renderer ---------------------------------------------
// tables [3R+1] float4: axis a, index i -> (a0, a3, a6, 0) of the per-axis recurrences (the
// same arithmetic as layer_tables_kernel), then (off3, 0, 0, 0).
__global__ void __launch_bounds__(kAxisThreads) separable_tables_kernel(const float *__restrict__ x0,
                                                                        const float *__restrict__ y1,
                                                                        const float *__restrict__ z2,
                                                                        const float *__restrict__ offset, uint32_t R,
                                                                        float4 *__restrict__ tables) {
    extern __shared__ float axis_s[];
    const int axis = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const float *a0 = axis == 0 ? x0 : (axis == 1 ? y1 : z2);
    float *s3 = axis_s + (size_t)2 * axis * R, *s6 = s3 + R;
    axis_recurrence(a0, offset[axis], R, lane, s3, s6);
    for (uint32_t i = lane; i < R; i += kWarp) tables[axis * R + i] = make_float4(a0[i], s3[i], s6[i], 0.0f);
    if (threadIdx.x == 0) tables[3 * R] = make_float4(offset[3], 0.0f, 0.0f, 0.0f);
}

// Adjoint (kernel/surface.cu:301-334 on the per-axis sums the fused renderer accumulated): the
// reverse recurrences over the table gradient (axis_reverse; 73 us at R = 256 as a chain of
// read-modify-writes in global memory, 8.0 us now), then the layer and offset gradients.
// offset[3]'s gradient is the sum of every cell's g6 = the x axis' a6 chain summed to index 0.
// The table gradient is consumed: it is left holding the recurrences' final values.
__global__ void __launch_bounds__(kAxisThreads) separable_grad_kernel(float4 *__restrict__ tg, uint32_t R,
                                                                      float *__restrict__ x_grad,
                                                                      float *__restrict__ y_grad,
                                                                      float *__restrict__ z_grad,
                                                                      float *__restrict__ offset_grad) {
    extern __shared__ float axis_s[];
    const int axis = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    float4 *t = tg + axis * R;  // (.x a0, .y a3, .z a6)
    float *g0 = axis_s + (size_t)3 * axis * R, *g3 = g0 + R, *g6 = g3 + R;
    for (uint32_t i = lane; i < R; i += kWarp) {
        const float4 v = t[i];
        g0[i] = v.x;
        g3[i] = v.y;
        g6[i] = v.z;
    }
    axis_reverse(g0, g3, g6, R, lane);
    float *out = axis == 0 ? x_grad : (axis == 1 ? y_grad : z_grad);
    for (uint32_t i = lane; i < R; i += kWarp) {
        out[i] = g0[i];
        t[i] = make_float4(g0[i], g3[i], g6[i], t[i].w);
    }
    if (lane == 0) {
        offset_grad[axis] = g3[0];
        if (axis == 0) offset_grad[3] = g6[0];
    }
}

// ---- SDF / normal samples ------------------------------------------------------------------

__device__ __forceinline__ bool cell_ok(int32_t idx, uint64_t cells) {
    if (idx < 0 || (uint64_t)idx >= cells) {
        flag_error(QSDVR_DEVERR_INDEX);
        return false;
    }
    return true;
}

// Gradient accumulation into a cell's 7 floats (the last one absent for a normal), no atomic for
// exact zeros (bit-identical: the accumulator starts at +0 and never holds -0; NaN and inf are
// still added).  A cell starts at a multiple of 28 bytes, so from an even cell on, or one float
// into an odd one, pairs are 8-byte aligned where the buffer is: 4 REDs instead of 7, which is
// what bounds the pass (1.3 M samples at 128^3: SDF backward
// 51 -> 39 us, normal backward 47 -> 38).
__device__ __forceinline__ void add_nonzero(float *p, float v) {
    if (v != 0.0f) atomicAdd(p, v);
}
__device__ __forceinline__ void add_nonzero2(float *p, float a, float b) {
    if (a != 0.0f || b != 0.0f) atomicAdd(reinterpret_cast<float2 *>(p), make_float2(a, b));
}
template <int kN>
__device__ __forceinline__ void add_cell(float *d, const float *g) {
    const uint32_t low = (uint32_t)(reinterpret_cast<uintptr_t>(d) & 7u);
    if (low == 0) {
#pragma unroll
        for (int k = 0; k + 1 < kN; k += 2) add_nonzero2(d + k, g[k], g[k + 1]);
        if (kN & 1) add_nonzero(d + kN - 1, g[kN - 1]);
    } else {
        add_nonzero(d, g[0]);
#pragma unroll
        for (int k = 1; k + 1 < kN; k += 2) add_nonzero2(d + k, g[k], g[k + 1]);
        if (!(kN & 1)) add_nonzero(d + kN - 1, g[kN - 1]);
    }
}

// kernel/surface.cu:54-72.
__global__ void __launch_bounds__(256) sdf_forward_kernel(float *__restrict__ out, const float *__restrict__ g,
                                                          const float *__restrict__ pts,
                                                          const int32_t *__restrict__ index, uint64_t n,
                                                          float reso, uint64_t cells) {
    const uint64_t id = blockIdx.x * 256ull + threadIdx.x;
    if (id >= n) return;
    const int32_t idx = index[id];
    if (!cell_ok(idx, cells)) {
        out[id] = 0.0f;
        return;
    }
    const float *c = g + (uint64_t)idx * 7;
    const float px = pts[3 * id], py = pts[3 * id + 1], pz = pts[3 * id + 2];
    const float a0 = c[0] * px, a1 = c[1] * py, a2 = c[2] * pz;
    const float a3 = c[3], a4 = c[4], a5 = c[5], a6 = c[6];
    const float nx = 2 * a0 + a3, ny = 2 * a1 + a4, nz = 2 * a2 + a5;
    out[id] = ((a0 + a3) * px + (a1 + a4) * py + (a2 + a5) * pz + a6) / sqrtf(nx * nx + ny * ny + nz * nz) / reso;
}

// kernel/surface.cu:74-102.
__global__ void __launch_bounds__(256) sdf_backward_kernel(const float *__restrict__ gout,
                                                           const float *__restrict__ g,
                                                           const float *__restrict__ pts,
                                                           const int32_t *__restrict__ index,
                                                           float *__restrict__ gg, uint64_t n, float reso,
                                                           uint64_t cells) {
    const uint64_t id = blockIdx.x * 256ull + threadIdx.x;
    if (id >= n) return;
    const int32_t idx = index[id];
    if (!cell_ok(idx, cells)) return;
    const float *c = g + (uint64_t)idx * 7;
    float *d = gg + (uint64_t)idx * 7;
    const float px = pts[3 * id], py = pts[3 * id + 1], pz = pts[3 * id + 2];
    const float a0 = c[0] * px, a1 = c[1] * py, a2 = c[2] * pz;
    const float a3 = c[3], a4 = c[4], a5 = c[5], a6 = c[6];
    const float value = (a0 + a3) * px + (a1 + a4) * py + (a2 + a5) * pz + a6;
    const float nx = 2 * a0 + a3, ny = 2 * a1 + a4, nz = 2 * a2 + a5;
    const float norm = 1.0f / sqrtf(nx * nx + ny * ny + nz * nz);
    const float norm3 = value * norm * norm * norm;
    const float go = gout[id] / reso;
    const float gr[7] = {go * px * (px * norm - 2 * nx * norm3), go * py * (py * norm - 2 * ny * norm3),
                         go * pz * (pz * norm - 2 * nz * norm3), go * (px * norm - nx * norm3),
                         go * (py * norm - ny * norm3),          go * (pz * norm - nz * norm3),
                         go * norm};
    add_cell<7>(d, gr);
}

// kernel/surface.cu:104-115.
__global__ void __launch_bounds__(256) normal_forward_kernel(float *__restrict__ out, const float *__restrict__ g,
                                                             const float *__restrict__ pts,
                                                             const int32_t *__restrict__ index, uint64_t n,
                                                             uint64_t cells) {
    const uint64_t id = blockIdx.x * 256ull + threadIdx.x;
    if (id >= n) return;
    const int32_t idx = index[id];
    if (!cell_ok(idx, cells)) {
        store3(out + 3 * id, f3{0.0f, 0.0f, 0.0f});
        return;
    }
    const float *c = g + (uint64_t)idx * 7;
    const float px = pts[3 * id], py = pts[3 * id + 1], pz = pts[3 * id + 2];
    const float vx = 2 * c[0] * px + c[3], vy = 2 * c[1] * py + c[4], vz = 2 * c[2] * pz + c[5];
    const float nrm = sqrtf(vx * vx + vy * vy + vz * vz);
    store3(out + 3 * id, f3{vx / nrm, vy / nrm, vz / nrm});
}

// kernel/surface.cu:117-146.
__global__ void __launch_bounds__(256) normal_backward_kernel(const float *__restrict__ gout,
                                                              const float *__restrict__ g,
                                                              const float *__restrict__ pts,
                                                              const int32_t *__restrict__ index,
                                                              float *__restrict__ gg, uint64_t n, uint64_t cells) {
    const uint64_t id = blockIdx.x * 256ull + threadIdx.x;
    if (id >= n) return;
    const int32_t idx = index[id];
    if (!cell_ok(idx, cells)) return;
    const float *c = g + (uint64_t)idx * 7;
    float *d = gg + (uint64_t)idx * 7;
    const float px = pts[3 * id], py = pts[3 * id + 1], pz = pts[3 * id + 2];
    const float a0 = 2 * c[0] * px, a1 = 2 * c[1] * py, a2 = 2 * c[2] * pz;
    const float a3 = c[3], a4 = c[4], a5 = c[5];
    const float vx = a0 + a3, vy = a1 + a4, vz = a2 + a5;
    const float norm = 1.0f / sqrtf(vx * vx + vy * vy + vz * vz);
    const float norm3 = norm * norm * norm;
    const float ox = gout[3 * id], oy = gout[3 * id + 1], oz = gout[3 * id + 2];
    const float gx = ox * (norm - norm3 * vx * vx) - oy * vy * norm3 * vx - oz * vz * norm3 * vx;
    const float gy = oy * (norm - norm3 * vy * vy) - ox * vx * norm3 * vy - oz * vz * norm3 * vy;
    const float gz = oz * (norm - norm3 * vz * vz) - oy * vy * norm3 * vz - ox * vx * norm3 * vz;
    const float gr[6] = {2.0f * px * gx, 2.0f * py * gy, 2.0f * pz * gz, gx, gy, gz};
    add_cell<6>(d, gr);
}

}  // namespace
}  // namespace qsdvr

using namespace qsdvr;

static constexpr uint32_t kMaxReso = 1290;  // (R+1)^3 * 32 floats must stay addressable

extern "C" size_t qsdvr_layer_to_grid_workspace_size(uint32_t reso) { return (size_t)6 * reso * sizeof(float); }

extern "C" int qsdvr_layer_to_grid_forward(float *grid7, const float *x_layer, const float *y_layer,
                                           const float *z_layer, const float *offset, uint32_t reso,
                                           void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    if (!grid7 || !x_layer || !y_layer || !z_layer || !offset)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_layer_to_grid_forward: null pointer");
    if (reso == 0 || reso > kMaxReso)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_layer_to_grid_forward: reso %u out of range", reso);
    if (!workspace || workspace_bytes < qsdvr_layer_to_grid_workspace_size(reso) || !aligned(workspace, 4))
        return set_error(QSDVR_ERR_WORKSPACE, "qsdvr_layer_to_grid_forward: workspace too small");
    float *tables = static_cast<float *>(workspace);
    layer_tables_kernel<<<1, kAxisThreads, axis_smem(reso, 2), stream>>>(x_layer, y_layer, z_layer, offset, reso,
                                                                        tables);
    const uint32_t rows = reso * reso;
    layer_expand_kernel<<<rows < 148u * 8 ? rows : 148u * 8, 256, (size_t)3 * reso * sizeof(float), stream>>>(
        grid7, x_layer, y_layer, z_layer, tables, offset, reso);
    return check_launch("qsdvr_layer_to_grid_forward");
}

extern "C" int qsdvr_layer_to_grid_backward(const float *grad7, uint32_t reso, float *x_grad, float *y_grad,
                                            float *z_grad, float *offset_grad, void *workspace,
                                            size_t workspace_bytes, cudaStream_t stream) {
    if (!grad7 || !x_grad || !y_grad || !z_grad || !offset_grad)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_layer_to_grid_backward: null pointer");
    if (reso == 0 || reso > kMaxReso)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_layer_to_grid_backward: reso %u out of range", reso);
    if (!workspace || workspace_bytes < qsdvr_layer_to_grid_workspace_size(reso) || !aligned(workspace, 4))
        return set_error(QSDVR_ERR_WORKSPACE, "qsdvr_layer_to_grid_backward: workspace too small");
    float *acc = static_cast<float *>(workspace);
    int st = check_cuda(cudaMemsetAsync(acc, 0, qsdvr_layer_to_grid_workspace_size(reso), stream), "memset");
    if (st == QSDVR_OK) st = check_cuda(cudaMemsetAsync(x_grad, 0, reso * sizeof(float), stream), "memset");
    if (st == QSDVR_OK) st = check_cuda(cudaMemsetAsync(y_grad, 0, reso * sizeof(float), stream), "memset");
    if (st == QSDVR_OK) st = check_cuda(cudaMemsetAsync(z_grad, 0, reso * sizeof(float), stream), "memset");
    if (st == QSDVR_OK) st = check_cuda(cudaMemsetAsync(offset_grad, 0, 4 * sizeof(float), stream), "memset");
    if (st != QSDVR_OK) return st;
    const uint32_t rows = reso * reso, per_block = (rows + kReduceBlocks - 1) / kReduceBlocks;
    const unsigned threads = reso >= 256 ? 256 : (reso + 31) / 32 * 32;
    layer_grad_reduce_kernel<<<(rows + per_block - 1) / per_block, threads, 3 * per_block * sizeof(float), stream>>>(
        grad7, reso, per_block, x_grad, y_grad, z_grad, acc, offset_grad + 3);
    layer_grad_reverse_kernel<<<1, kAxisThreads, axis_smem(reso, 3), stream>>>(x_grad, y_grad, z_grad, acc,
                                                                              offset_grad, reso);
    return check_launch("qsdvr_layer_to_grid_backward");
}

extern "C" int qsdvr_separable_sdf_tables(const float *x_layer, const float *y_layer, const float *z_layer,
                                          const float *offset, uint32_t reso, float *tables, cudaStream_t stream) {
    if (!x_layer || !y_layer || !z_layer || !offset || !tables)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_separable_sdf_tables: null pointer");
    if (reso == 0 || reso > kMaxReso)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_separable_sdf_tables: reso %u out of range", reso);
    if (!aligned(tables, 16)) return set_error(QSDVR_ERR_ALIGNMENT, "qsdvr_separable_sdf_tables: tables alignment");
    separable_tables_kernel<<<1, kAxisThreads, axis_smem(reso, 2), stream>>>(x_layer, y_layer, z_layer, offset, reso,
                                                                            reinterpret_cast<float4 *>(tables));
    return check_launch("qsdvr_separable_sdf_tables");
}

extern "C" int qsdvr_separable_sdf_grad(float *table_grad, uint32_t reso, float *x_grad, float *y_grad,
                                        float *z_grad, float *offset_grad, cudaStream_t stream) {
    if (!table_grad || !x_grad || !y_grad || !z_grad || !offset_grad)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_separable_sdf_grad: null pointer");
    if (reso == 0 || reso > kMaxReso)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_separable_sdf_grad: reso %u out of range", reso);
    if (!aligned(table_grad, 16)) return set_error(QSDVR_ERR_ALIGNMENT, "qsdvr_separable_sdf_grad: alignment");
    separable_grad_kernel<<<1, kAxisThreads, axis_smem(reso, 3), stream>>>(reinterpret_cast<float4 *>(table_grad), reso,
                                                                          x_grad, y_grad, z_grad, offset_grad);
    return check_launch("qsdvr_separable_sdf_grad");
}

extern "C" int qsdvr_sample_sdf_forward(float *out, const float *grid7, const float *points, const int32_t *index,
                                        uint64_t count, float reso, uint64_t cell_count, cudaStream_t stream) {
    if (count == 0) return QSDVR_OK;
    if (!out || !grid7 || !points || !index)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_sample_sdf_forward: null pointer");
    sdf_forward_kernel<<<grid_for(count, 256), 256, 0, stream>>>(out, grid7, points, index, count, reso, cell_count);
    return check_launch("qsdvr_sample_sdf_forward");
}

extern "C" int qsdvr_sample_sdf_backward(const float *grad_out, const float *grid7, const float *points,
                                         const int32_t *index, float *grid7_grad, uint64_t count, float reso,
                                         uint64_t cell_count, cudaStream_t stream) {
    if (count == 0) return QSDVR_OK;
    if (!grad_out || !grid7 || !points || !index || !grid7_grad)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_sample_sdf_backward: null pointer");
    sdf_backward_kernel<<<grid_for(count, 256), 256, 0, stream>>>(grad_out, grid7, points, index, grid7_grad, count,
                                                                  reso, cell_count);
    return check_launch("qsdvr_sample_sdf_backward");
}

extern "C" int qsdvr_sample_normal_forward(float *out, const float *grid7, const float *points,
                                           const int32_t *index, uint64_t count, uint64_t cell_count,
                                           cudaStream_t stream) {
    if (count == 0) return QSDVR_OK;
    if (!out || !grid7 || !points || !index)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_sample_normal_forward: null pointer");
    normal_forward_kernel<<<grid_for(count, 256), 256, 0, stream>>>(out, grid7, points, index, count, cell_count);
    return check_launch("qsdvr_sample_normal_forward");
}

extern "C" int qsdvr_sample_normal_backward(const float *grad_out, const float *grid7, const float *points,
                                            const int32_t *index, float *grid7_grad, uint64_t count,
                                            uint64_t cell_count, cudaStream_t stream) {
    if (count == 0) return QSDVR_OK;
    if (!grad_out || !grid7 || !points || !index || !grid7_grad)
        return set_error(QSDVR_ERR_INVALID_ARGUMENT, "qsdvr_sample_normal_backward: null pointer");
    normal_backward_kernel<<<grid_for(count, 256), 256, 0, stream>>>(grad_out, grid7, points, index, grid7_grad,
                                                                     count, cell_count);
    return check_launch("qsdvr_sample_normal_backward");
}
