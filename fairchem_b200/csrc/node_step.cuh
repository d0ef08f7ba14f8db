// Node-wise and radial kernels of the whole-model evaluation (fcb200_model_forward / _backward): residual add + RMS norm
// in one pass, hidden activations of all radial MLPs at once, system embedding, energy sum and the start of the
// backward pass.  All are one pass over their tensors (HBM-bound at size, launch-bound when small).
#pragma once

#include "step.cuh"
#include "shape_lx.cuh"

namespace fcb200 {
namespace step {

__host__ __device__ constexpr int degree_of(int L) {
    int l = 0;
    while ((l + 1) * (l + 1) <= L) ++l;
    return l;
}
template <int LMAX> __host__ __device__ constexpr float balance_of(int L) {
    return 1.0f / (float)((2 * degree_of(L) + 1) * (LMAX + 1));
}
__device__ __forceinline__ float hsum4(float4 v) { return v.x + v.y + v.z + v.w; }
__device__ __forceinline__ float sigm(float v) { return 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ float dsilu(float v) {
    const float s = sigm(v);
    return s * (1.0f + v * (1.0f - s));
}
__device__ __forceinline__ float max4(float m, float4 v) {
    return fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
}

// every thread of the block calls this once with its largest |value|
__device__ __forceinline__ void report_max(Scale* s, float m) {
    __shared__ float sm[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(kFull, m, o));
    if (lane == 0) sm[wid] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i) m = fmaxf(m, sm[i]);
        atomicMax(&s->amax, __float_as_uint(m));
        __threadfence();
        if (atomicAdd(&s->ticket, 1u) == gridDim.x - 1) {
            __threadfence();
            const float a = __uint_as_float(atomicMax(&s->amax, 0u));
            s->scale = exp2f(floorf(6.0f - log2f(fmaxf(a, 1e-30f))));
        }
    }
}

// x = a (+ b); out = norm(x) * weight (+ bias + system embedding on row 0).  One warp per node, the node's rows stay in
// registers between the statistics and the output: one read and one write per tensor.  Memory-bound: 100 000 nodes of lmax 2,
// 5.8 -> 6.1 TB/s with the residual, the planes and the system embedding in the same pass (three passes before).
// sum: where x goes when b is given.  out_f32 / planes: either may be absent.  row0: half planes of row 0 of the output.
template <int LMAX>
__global__ void __launch_bounds__(128)
    norm_fwd_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ sum,
                    const float* __restrict__ weight, const float* __restrict__ bias, const float* __restrict__ sys,
                    const int32_t* __restrict__ batch, float* __restrict__ out_f32, OutSplit planes, OutSplit row0,
                    float* __restrict__ stats, float eps, int64_t num_nodes) {
    pdl_sync();
    constexpr int kL = (LMAX + 1) * (LMAX + 1);
    planes.s = row0.s = 1.0f;
    const int lane = threadIdx.x & 31, c = lane * 4;
    for (int64_t n = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); n < num_nodes; n += (int64_t)gridDim.x * 4) {
        const int64_t o = n * kL * C + c;
        float4 x[kL];
#pragma unroll
        for (int L = 0; L < kL; ++L) x[L] = ld4(a + o + L * C);
        if (b) {
#pragma unroll
            for (int L = 0; L < kL; ++L) x[L] = add4(x[L], ld4(b + o + L * C));
#pragma unroll
            for (int L = 0; L < kL; ++L) st4(sum + o + L * C, x[L]);
        }
        const float mean0 = warp_sum(hsum4(x[0])) * (1.0f / C);
        x[0] = make_float4(x[0].x - mean0, x[0].y - mean0, x[0].z - mean0, x[0].w - mean0);
        float acc = 0.f;
#pragma unroll
        for (int L = 0; L < kL; ++L) acc = fmaf(balance_of<LMAX>(L), dot4(x[L], x[L]), acc);
        const float scale = rsqrtf(warp_sum(acc) * (1.0f / C) + eps);
#pragma unroll
        for (int L = 0; L < kL; ++L) {
            float4 v = mul4(scale4(scale, x[L]), ld4(weight + degree_of(L) * C + c));
            if (L == 0) {
                v = add4(v, ld4(bias + c));
                if (sys) v = add4(v, ld4(sys + (int64_t)batch[n] * C + c));
                if (row0.hi) row0.st(n * C + c, v);
            }
            if (out_f32) st4(out_f32 + o + L * C, v);
            if (planes.hi) planes.st(o + L * C, v);
        }
        if (lane == 0) {
            stats[n * 2 + 0] = mean0;
            stats[n * 2 + 1] = scale;
        }
    }
}

// Memory-bound: 100 000 nodes of lmax 2, 4.2 -> 6.6 TB/s, the residual's gradient and the largest value in the same pass.
// lmax 4 holds 25 rows twice in 255 registers and spills 40 bytes; 20 000 nodes 5.9 TB/s.
// grad_x = residual + d norm; g has all rows, or (ROW0) only row 0 of every node, [N, C]
template <int LMAX, bool ROW0>
__global__ void __launch_bounds__(128)
    norm_bwd_kernel(const float* __restrict__ g, const float* __restrict__ x, const float* __restrict__ weight,
                    const float* __restrict__ stats, const float* __restrict__ residual, float* __restrict__ grad_x,
                    Scale* __restrict__ scale_out, int64_t num_nodes) {
    pdl_sync();
    constexpr int kL = (LMAX + 1) * (LMAX + 1);
    const int lane = threadIdx.x & 31, c = lane * 4;
    float amax = 0.f;
    for (int64_t n = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); n < num_nodes; n += (int64_t)gridDim.x * 4) {
        const int64_t o = n * kL * C + c;
        const float mean0 = stats[n * 2 + 0], scale = stats[n * 2 + 1];
        float4 v[kL], gw[ROW0 ? 1 : kL];
#pragma unroll
        for (int L = 0; L < kL; ++L) v[L] = ld4(x + o + L * C);
#pragma unroll
        for (int L = 0; L < (ROW0 ? 1 : kL); ++L) gw[L] = mul4(ld4(g + (ROW0 ? n * C + c : o + L * C)), ld4(weight + degree_of(L) * C + c));
        v[0] = make_float4(v[0].x - mean0, v[0].y - mean0, v[0].z - mean0, v[0].w - mean0);
        float ds = 0.f;
#pragma unroll
        for (int L = 0; L < (ROW0 ? 1 : kL); ++L) ds += dot4(gw[L], v[L]);
        ds = warp_sum(ds);
        const float g0w = warp_sum(hsum4(gw[0])), y0b = warp_sum(hsum4(v[0]));
        const float k = scale * scale * scale * ds * (1.0f / C);
        const float mean_dy0 = (g0w * scale - k * balance_of<LMAX>(0) * y0b) * (1.0f / C);
#pragma unroll
        for (int L = 0; L < kL; ++L) {
            const float kb = -k * balance_of<LMAX>(L);
            float4 d = scale4(kb, v[L]);
            if (L == 0 || !ROW0) d = fma4(scale, gw[ROW0 ? 0 : L], d);
            if (L == 0) d = make_float4(d.x - mean_dy0, d.y - mean_dy0, d.z - mean_dy0, d.w - mean_dy0);
            if (residual) d = add4(d, ld4(residual + o + L * C));
            st4(grad_x + o + L * C, d);
            amax = max4(amax, d);
        }
    }
    report_max(scale_out, amax);
}

// half planes of a float32 tensor times a device scale; memory-bound, 5.6 TB/s at 100 000 nodes
__global__ void __launch_bounds__(256)
    split_kernel(const float* __restrict__ in, OutSplit out, const float* __restrict__ scale_ptr, int64_t quads) {
    pdl_sync();
    out.load_scale(scale_ptr);
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < quads; i += (int64_t)gridDim.x * 256) out.st(i * 4, ld4(in + i * 4));
}

// ---- hidden activations of the radial MLPs ------------------------------------------------------------------------
// SiLU(LayerNorm(pre + element tables)) for `nets` MLPs side by side.  Rows (edge, net) of 128: pre [E, nets*C], stats
// [E, nets, 2]; output planes out_row apart.  A warp takes R rows that follow one another, whatever edges they belong to.
// Bound by instruction issue (exponential, division, reductions), which the backward pass needs warps for and the forward
// pass independent rows: 1.55 M edges x 5 nets, ms, backward with 4 rows / 3 blocks on an SM 7.2, 4 / 4 6.6, 2 / 4 6.5, 2 / 5
// 6.2, 1 / 8 6.0; forward with 1 / 8 5.4, 2 / 5 5.4, 4 / 5 4.9.  One edge's nets three at a time, a sixth of the slots empty
// at five nets: 7.8 and 5.6.
constexpr int kRadialFwdRows = 4, kRadialBwdRows = 1;

inline int64_t radial_items(int64_t edges, int nets, int rows) { return (edges * nets + rows - 1) / rows; }

// rows [row0, row0 + n) of the pre-activation, tables added, and the nets they belong to
template <int R>
__device__ __forceinline__ void radial_rows(float4 (&y)[R], int (&net)[R], uint32_t row0, int n, const float* __restrict__ pre,
                                            const float* __restrict__ ts, const float* __restrict__ tt, const int32_t* __restrict__ z,
                                            const int32_t* __restrict__ src, const int32_t* __restrict__ tgt, int nets, int c) {
    uint32_t i = row0 / (uint32_t)nets;
    net[0] = (int)(row0 - i * nets);
#pragma unroll
    for (int b = 0; b < R; ++b) {
        if (b > 0) {
            const bool next = net[b - 1] + 1 == nets;
            net[b] = next ? 0 : net[b - 1] + 1;
            i += next ? 1 : 0;
        }
        y[b] = f4zero();
        if (b >= n) continue;
        y[b] = ld4(pre + (int64_t)(row0 + b) * C + c);
        if (ts) {
            const int64_t col = net[b] * C + c, width = (int64_t)nets * C;
            y[b] = add4(y[b], add4(ld4(ts + z[src[i]] * width + col), ld4(tt + z[tgt[i]] * width + col)));
        }
    }
}

__global__ void __launch_bounds__(256)
    radial_fwd_kernel(const float* __restrict__ pre, const float* __restrict__ ts, const float* __restrict__ tt,
                      const int32_t* __restrict__ z, const int32_t* __restrict__ src, const int32_t* __restrict__ tgt,
                      const float* __restrict__ gamma, const float* __restrict__ beta, float eps, OutSplit out, int64_t out_row,
                      float* __restrict__ stats, uint32_t rows, int nets) {
    pdl_sync();
    constexpr int R = kRadialFwdRows;
    out.s = 1.0f;
    const int lane = threadIdx.x & 31, c = lane * 4;
    for (uint32_t row0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * R; row0 < rows; row0 += gridDim.x * 8 * R) {
        const int n = min((uint32_t)R, rows - row0);
        float4 y[R];
        int net[R];
        radial_rows(y, net, row0, n, pre, ts, tt, z, src, tgt, nets, c);
        float mean[R], rstd[R];
#pragma unroll
        for (int b = 0; b < R; ++b) mean[b] = hsum4(y[b]);
        warp_sums(mean, lane);
#pragma unroll
        for (int b = 0; b < R; ++b) {
            mean[b] *= 1.0f / C;
            y[b] = make_float4(y[b].x - mean[b], y[b].y - mean[b], y[b].z - mean[b], y[b].w - mean[b]);
            rstd[b] = dot4(y[b], y[b]);
        }
        warp_sums(rstd, lane);
#pragma unroll
        for (int b = 0; b < R; ++b) {
            if (b >= n) break;
            rstd[b] = rsqrtf(rstd[b] * (1.0f / C) + eps);
            const int col = net[b] * C + c;
            const float4 gm = ld4(gamma + col), bt = ld4(beta + col), d = y[b];
            const float4 v = make_float4(fmaf(d.x * rstd[b], gm.x, bt.x), fmaf(d.y * rstd[b], gm.y, bt.y), fmaf(d.z * rstd[b], gm.z, bt.z),
                                         fmaf(d.w * rstd[b], gm.w, bt.w));
            out.st((row0 + b) * out_row + c, make_float4(v.x * sigm(v.x), v.y * sigm(v.y), v.z * sigm(v.z), v.w * sigm(v.w)));
            if (lane == 0) *reinterpret_cast<float2*>(stats + (int64_t)(row0 + b) * 2) = make_float2(mean[b], rstd[b]);
        }
    }
}

// backward of the same; the planes are written with the smallest of the nets' gradient scales (block 0 leaves it at
// scale_out), so that one contraction may sum over the nets
__global__ void __launch_bounds__(256, 8)
    radial_bwd_kernel(const float* __restrict__ grad_out, const float* __restrict__ pre, const float* __restrict__ ts,
                      const float* __restrict__ tt, const int32_t* __restrict__ z, const int32_t* __restrict__ src,
                      const int32_t* __restrict__ tgt, const float* __restrict__ gamma, const float* __restrict__ beta,
                      const float* __restrict__ stats, OutSplit out, int64_t out_row, const Scale* __restrict__ scales,
                      int num_scales, float* __restrict__ scale_out, uint32_t rows, int nets) {
    pdl_sync();
    constexpr int R = kRadialBwdRows;
    float s = scales[0].scale;
    for (int i = 1; i < num_scales; ++i) s = fminf(s, scales[i].scale);
    out.s = s;
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale_out = s;
    const int lane = threadIdx.x & 31, c = lane * 4;
    for (uint32_t row0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * R; row0 < rows; row0 += gridDim.x * 8 * R) {
        const int n = min((uint32_t)R, rows - row0);
        float4 y[R], go[R];
        float2 st[R];
        int net[R];
#pragma unroll
        for (int b = 0; b < R; ++b) {
            go[b] = b < n ? ld4(grad_out + (int64_t)(row0 + b) * C + c) : f4zero();
            st[b] = b < n ? *reinterpret_cast<const float2*>(stats + (int64_t)(row0 + b) * 2) : make_float2(0.f, 0.f);
        }
        radial_rows(y, net, row0, n, pre, ts, tt, z, src, tgt, nets, c);
        float sum[2 * R];
#pragma unroll
        for (int b = 0; b < R; ++b) {
            const int col = net[b] * C + c;
            const float4 gm = ld4(gamma + col), bt = ld4(beta + col);
            const float4 xh = make_float4((y[b].x - st[b].x) * st[b].y, (y[b].y - st[b].x) * st[b].y, (y[b].z - st[b].x) * st[b].y, (y[b].w - st[b].x) * st[b].y);
            go[b] = make_float4(go[b].x * dsilu(fmaf(xh.x, gm.x, bt.x)) * gm.x, go[b].y * dsilu(fmaf(xh.y, gm.y, bt.y)) * gm.y,
                                go[b].z * dsilu(fmaf(xh.z, gm.z, bt.z)) * gm.z, go[b].w * dsilu(fmaf(xh.w, gm.w, bt.w)) * gm.w);
            y[b] = xh;
            sum[b] = hsum4(go[b]);
            sum[R + b] = dot4(go[b], xh);
        }
        warp_sums(sum, lane);
#pragma unroll
        for (int b = 0; b < R; ++b) {
            if (b >= n) break;
            const float s1 = sum[b] * (1.0f / C), s2 = sum[R + b] * (1.0f / C);
            out.st((row0 + b) * out_row + c, make_float4(st[b].y * (go[b].x - s1 - y[b].x * s2), st[b].y * (go[b].y - s1 - y[b].y * s2),
                                                         st[b].y * (go[b].z - s1 - y[b].z * s2), st[b].y * (go[b].w - s1 - y[b].w * s2)));
        }
    }
}

// ---- system embedding: silu(W [charge | spin | dataset] + b), one block per system ----------------------------------
// Eight threads share an output channel, 48 of the 384 products each: one system is a latency chain (384 dependent
// multiply-adds behind their weight loads took 25 us).
__global__ void __launch_bounds__(8 * C)
    system_kernel(const int64_t* __restrict__ charge, const int64_t* __restrict__ spin, const int32_t* __restrict__ dataset,
                  const float* __restrict__ charge_emb, const float* __restrict__ spin_emb, const float* __restrict__ dataset_emb,
                  const float* __restrict__ w_t, const float* __restrict__ bias, float* __restrict__ out, int32_t* __restrict__ status) {
    pdl_sync();
    __shared__ float part[8][C];
    const int s = blockIdx.x, c = threadIdx.x & (C - 1), p = threadIdx.x / C;
    int64_t q = charge[s] + 100, m = spin[s];
    if (q < 0 || q > 200 || m < 0 || m > 100) {  // outside the embedding tables: report, do not read
        if (threadIdx.x == 0) atomicExch(status, 3);
        q = m = 0;
    }
    const float* rows[3] = {charge_emb + q * C, spin_emb + m * C, dataset_emb + (int64_t)dataset[s] * C};
    float acc = 0.f;
#pragma unroll 16
    for (int j = 0; j < 48; ++j) {
        const int k = p * 48 + j;
        acc = fmaf(__ldg(rows[k / C] + k % C), __ldg(w_t + k * C + c), acc);
    }
    part[p][c] = acc;
    __syncthreads();
    if (p) return;
    acc = bias[c];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc += part[i][c];
    out[s * C + c] = acc * sigm(acc);
}

// ---- energy head -----------------------------------------------------------------------------------------------------
// energy[batch[n]] += silu(y[n]) . w + b in float64, node rows [N, C]; one warp per node, a warp's consecutive nodes are
// summed before the atomic add (systems are contiguous in the batch)
__global__ void __launch_bounds__(256)
    energy_kernel(const float* __restrict__ y, const float* __restrict__ w, const float* __restrict__ b, const int32_t* __restrict__ batch,
                  double* __restrict__ energy, int64_t num_nodes, int per_warp) {
    pdl_sync();
    const int lane = threadIdx.x & 31, c = lane * 4;
    const int64_t n0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * per_warp;
    const float4 wv = ld4(w + c);
    double sum = 0.0;
    int cur = -1;
    for (int64_t n = n0; n < n0 + per_warp && n < num_nodes; ++n) {
        const float4 v = ld4(y + n * C + c);
        const float e = warp_sum(v.x * sigm(v.x) * wv.x + v.y * sigm(v.y) * wv.y + v.z * sigm(v.z) * wv.z + v.w * sigm(v.w) * wv.w) + b[0];
        const int s = batch[n];
        if (s != cur) {
            if (cur >= 0 && lane == 0) atomicAdd(energy + cur, sum);
            cur = s;
            sum = 0.0;
        }
        sum += (double)e;
    }
    if (cur >= 0 && lane == 0) atomicAdd(energy + cur, sum);
}

// gradient of every node's energy with respect to the last hidden pre-activation, as half planes
__global__ void __launch_bounds__(256)
    energy_bwd_kernel(const float* __restrict__ y, const float* __restrict__ w, OutSplit out, const float* __restrict__ scale_ptr,
                      int64_t num_nodes) {
    pdl_sync();
    out.load_scale(scale_ptr);
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < num_nodes * (C / 4); i += (int64_t)gridDim.x * 256) {
        const float4 v = ld4(y + i * 4), wv = ld4(w + (i % (C / 4)) * 4);
        out.st(i * 4, make_float4(wv.x * dsilu(v.x), wv.y * dsilu(v.y), wv.z * dsilu(v.z), wv.w * dsilu(v.w)));
    }
}

// sum over the edges of grad_vec (x) vec per system (the strain derivative), float64
__global__ void __launch_bounds__(256)
    virial_kernel(const float* __restrict__ grad_vec, const float4* __restrict__ vec, const int32_t* __restrict__ tgt,
                  const int32_t* __restrict__ batch, double* __restrict__ virial, int64_t num_edges, int per_warp) {
    pdl_sync();
    const int lane = threadIdx.x & 31;
    const int64_t w0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * per_warp;
    const int i = lane / 3, j = lane % 3;  // lanes 0..8 own one component each
    double sum = 0.0;
    int cur = -1;
    for (int64_t e = w0; e < w0 + per_warp && e < num_edges; ++e) {
        const int s = batch[tgt[e]];
        if (s != cur) {
            if (cur >= 0 && lane < 9) atomicAdd(virial + cur * 9 + lane, sum);
            cur = s;
            sum = 0.0;
        }
        if (lane < 9) sum += (double)grad_vec[e * 3 + i] * (double)(reinterpret_cast<const float*>(vec + e)[j]);
    }
    if (cur >= 0 && lane < 9) atomicAdd(virial + cur * 9 + lane, sum);
}

}  // namespace step
}  // namespace fcb200
