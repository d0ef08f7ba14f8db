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
// SiLU(LayerNorm(pre + element tables)) for `nets` MLPs side by side.  Rows: pre [E, nets*C], stats [E, nets, 2]; output
// planes at i * out_ld + net * out_net.  One warp per edge and kNetBatch nets: one row of 512 bytes per warp left the
// loads and the two reductions of a row in series (3.1 M edges x 5 nets: 10.8 ms forward, 14.0 ms backward).
constexpr int kNetBatch = 3;

struct RadialItem {
    int64_t i;
    int net0, n;
};
__device__ __forceinline__ RadialItem radial_item(int64_t it, int nets) {
    const int groups = (nets + kNetBatch - 1) / kNetBatch;
    const int64_t i = it / groups;
    const int net0 = (int)(it - i * groups) * kNetBatch;
    return {i, net0, min(kNetBatch, nets - net0)};
}
__host__ __device__ inline int64_t radial_items(int64_t edges, int nets) { return edges * ((nets + kNetBatch - 1) / kNetBatch); }

__device__ __forceinline__ void radial_rows(float4 (&y)[kNetBatch], const RadialItem& q, const float* __restrict__ pre, const float* __restrict__ ts,
                                            const float* __restrict__ tt, const int32_t* __restrict__ z, const int32_t* __restrict__ src,
                                            const int32_t* __restrict__ tgt, int64_t e_base, int64_t width, int c) {
#pragma unroll
    for (int b = 0; b < kNetBatch; ++b) y[b] = b < q.n ? ld4(pre + q.i * width + (q.net0 + b) * C + c) : f4zero();
    if (ts) {
        const float* s0 = ts + z[src[e_base + q.i]] * width + q.net0 * C + c;
        const float* t0 = tt + z[tgt[e_base + q.i]] * width + q.net0 * C + c;
#pragma unroll
        for (int b = 0; b < kNetBatch; ++b)
            if (b < q.n) y[b] = add4(y[b], add4(ld4(s0 + b * C), ld4(t0 + b * C)));
    }
}

__global__ void __launch_bounds__(256)
    radial_fwd_kernel(const float* __restrict__ pre, const float* __restrict__ ts, const float* __restrict__ tt,
                      const int32_t* __restrict__ z, const int32_t* __restrict__ src, const int32_t* __restrict__ tgt,
                      const float* __restrict__ gamma, const float* __restrict__ beta, float eps, OutSplit out, int64_t out_ld,
                      int out_net, float* __restrict__ stats, int64_t e_base, int64_t num_edges, int nets) {
    pdl_sync();
    out.s = 1.0f;
    const int lane = threadIdx.x & 31, c = lane * 4;
    const int64_t items = radial_items(num_edges, nets), width = (int64_t)nets * C;
    for (int64_t it = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); it < items; it += (int64_t)gridDim.x * 8) {
        const RadialItem q = radial_item(it, nets);
        float4 y[kNetBatch];
        radial_rows(y, q, pre, ts, tt, z, src, tgt, e_base, width, c);
        float mean[kNetBatch], rstd[kNetBatch];
#pragma unroll
        for (int b = 0; b < kNetBatch; ++b) mean[b] = warp_sum(hsum4(y[b])) * (1.0f / C);
#pragma unroll
        for (int b = 0; b < kNetBatch; ++b) {
            y[b] = make_float4(y[b].x - mean[b], y[b].y - mean[b], y[b].z - mean[b], y[b].w - mean[b]);
            rstd[b] = rsqrtf(warp_sum(dot4(y[b], y[b])) * (1.0f / C) + eps);
        }
#pragma unroll
        for (int b = 0; b < kNetBatch; ++b) {
            if (b >= q.n) break;
            const int col = (q.net0 + b) * C + c;
            const float4 gm = ld4(gamma + col), bt = ld4(beta + col), d = y[b];
            const float4 v = make_float4(fmaf(d.x * rstd[b], gm.x, bt.x), fmaf(d.y * rstd[b], gm.y, bt.y), fmaf(d.z * rstd[b], gm.z, bt.z),
                                         fmaf(d.w * rstd[b], gm.w, bt.w));
            out.st(q.i * out_ld + (q.net0 + b) * out_net + c, make_float4(v.x * sigm(v.x), v.y * sigm(v.y), v.z * sigm(v.z), v.w * sigm(v.w)));
            if (lane == 0) *reinterpret_cast<float2*>(stats + (q.i * nets + q.net0 + b) * 2) = make_float2(mean[b], rstd[b]);
        }
    }
}

// backward of the same; the planes are written with the smallest of the nets' gradient scales (block 0 leaves it at
// scale_out), so that one contraction may sum over the nets
__global__ void __launch_bounds__(256)
    radial_bwd_kernel(const float* __restrict__ grad_out, const float* __restrict__ pre, const float* __restrict__ ts,
                      const float* __restrict__ tt, const int32_t* __restrict__ z, const int32_t* __restrict__ src,
                      const int32_t* __restrict__ tgt, const float* __restrict__ gamma, const float* __restrict__ beta,
                      const float* __restrict__ stats, OutSplit out, int64_t out_ld, int out_net, const Scale* __restrict__ scales,
                      int num_scales, float* __restrict__ scale_out, int64_t e_base, int64_t num_edges, int nets) {
    pdl_sync();
    float s = scales[0].scale;
    for (int i = 1; i < num_scales; ++i) s = fminf(s, scales[i].scale);
    out.s = s;
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale_out = s;
    const int lane = threadIdx.x & 31, c = lane * 4;
    const int64_t items = radial_items(num_edges, nets), width = (int64_t)nets * C;
    for (int64_t it = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); it < items; it += (int64_t)gridDim.x * 8) {
        const RadialItem q = radial_item(it, nets);
        float4 y[kNetBatch], go[kNetBatch];
        float2 st[kNetBatch];
#pragma unroll
        for (int b = 0; b < kNetBatch; ++b) {
            go[b] = b < q.n ? ld4(grad_out + q.i * width + (q.net0 + b) * C + c) : f4zero();
            st[b] = b < q.n ? *reinterpret_cast<const float2*>(stats + (q.i * nets + q.net0 + b) * 2) : make_float2(0.f, 0.f);
        }
        radial_rows(y, q, pre, ts, tt, z, src, tgt, e_base, width, c);
        float s1[kNetBatch], s2[kNetBatch];
#pragma unroll
        for (int b = 0; b < kNetBatch; ++b) {
            const int col = (q.net0 + (b < q.n ? b : 0)) * C + c;
            const float4 gm = ld4(gamma + col), bt = ld4(beta + col);
            const float4 xh = make_float4((y[b].x - st[b].x) * st[b].y, (y[b].y - st[b].x) * st[b].y, (y[b].z - st[b].x) * st[b].y, (y[b].w - st[b].x) * st[b].y);
            go[b] = make_float4(go[b].x * dsilu(fmaf(xh.x, gm.x, bt.x)) * gm.x, go[b].y * dsilu(fmaf(xh.y, gm.y, bt.y)) * gm.y,
                                go[b].z * dsilu(fmaf(xh.z, gm.z, bt.z)) * gm.z, go[b].w * dsilu(fmaf(xh.w, gm.w, bt.w)) * gm.w);
            y[b] = xh;
            s1[b] = warp_sum(hsum4(go[b])) * (1.0f / C);
            s2[b] = warp_sum(dot4(go[b], xh)) * (1.0f / C);
        }
#pragma unroll
        for (int b = 0; b < kNetBatch; ++b) {
            if (b >= q.n) break;
            out.st(q.i * out_ld + (q.net0 + b) * out_net + c,
                   make_float4(st[b].y * (go[b].x - s1[b] - y[b].x * s2[b]), st[b].y * (go[b].y - s1[b] - y[b].y * s2[b]),
                               st[b].y * (go[b].z - s1[b] - y[b].z * s2[b]), st[b].y * (go[b].w - s1[b] - y[b].w * s2[b])));
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
