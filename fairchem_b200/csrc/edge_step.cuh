// Edge kernels of the whole-model evaluation (fcb200_model_forward / _backward), for lmax = 2 and 4 with mmax = 2.
//
// Forward they compute what edge_geometry.cu and edge_block*.cu do, with the envelope applied while the Wigner block is
// staged (no inverse tensor).  The backward pass differs: the gradient with respect to the Wigner entries of an edge
// (35 or 115 numbers) is never formed.  A rotation has three degrees of freedom, so the entries matter only through
// the torque
//     tau_a = d loss / d theta_a   under   D -> D exp(theta . G),        G_a = the rotation generators of degree l,
// and for a gathered row x with rotated-back gradient g = D^T grad this is sum_ij g_i (G_a)_ij x_j: a handful of
// products with vectors the kernel already holds, and three numbers to reduce over a warp instead of 35.  The edge
// frame R takes the edge vector v to +Y and the network does not depend on the roll about it, hence
// d loss / d v (perpendicular part) = (v x tau) / |v|^2.
//
// One warp works on one edge (or on the edges of one node in turn); a lane owns 4 of the 128 channels.  Sums over the
// edges of a node have a fixed order, no atomics.
#pragma once

#include "common.cuh"
#include "geometry.cuh"
#include "shape_lx.cuh"
#include "step.cuh"

namespace fcb200 {
namespace step {

// ---- generators -----------------------------------------------------------------------------------------------
// Real harmonics with the y axis as the pole, index m + l.  Upper triangle of the antisymmetric G_a:
//   G_y[-m, m] = m;   G_x[0, 1] = G_z[-1, 0] = -sqrt(l(l+1)/2);   with c = sqrt((l-m)(l+m+1)) / 2 for m >= 1:
//   G_x[-m-1, -m] = c, G_x[m, m+1] = -c, G_z[-m-1, m] = G_z[-m, m+1] = -c.
template <int l, int m, class P>
__device__ __forceinline__ void torque_pairs(P&& pr, float (&t)[3]) {
    constexpr float c = (float)(0.5 * csqrt((double)(l - m) * (l + m + 1)));
    t[0] = fmaf(c, pr(l - m - 1, l - m) - pr(l + m, l + m + 1), t[0]);
    t[2] = fmaf(-c, pr(l - m - 1, l + m) + pr(l - m, l + m + 1), t[2]);
    if constexpr (m + 1 < l) torque_pairs<l, m + 1>(pr, t);
}
// t_a += sum_{i<j} G_a[i, j] (g_i x_j - g_j x_i)
template <int l>
__device__ __forceinline__ void torque(const float4 (&g)[2 * l + 1], const float4 (&x)[2 * l + 1], float (&t)[3]) {
    if constexpr (l > 0) {
        auto pr = [&](int i, int j) { return dot4(g[i], x[j]) - dot4(g[j], x[i]); };
#pragma unroll
        for (int m = 1; m <= l; ++m) t[1] = fmaf((float)m, pr(l - m, l + m), t[1]);
        constexpr float s0 = (float)csqrt(0.5 * l * (l + 1));
        t[0] = fmaf(-s0, pr(l, l + 1), t[0]);
        t[2] = fmaf(-s0, pr(l - 1, l), t[2]);
        if constexpr (l >= 2) torque_pairs<l, 1>(pr, t);
    }
}

// sum of 4 per-lane values over the warp; lane i (i < 4) returns total i.  Two exchange steps that halve the number
// of values, then three plain steps: 6 shuffles instead of 20.
__device__ __forceinline__ float reduce4(float a, float b, float c, float d, int lane) {
    const bool up = lane & 1;
    float p = (up ? b : a) + __shfl_xor_sync(kFull, up ? a : b, 1);
    float q = (up ? d : c) + __shfl_xor_sync(kFull, up ? c : d, 1);
    const bool up2 = lane & 2;
    float r = (up2 ? q : p) + __shfl_xor_sync(kFull, up2 ? p : q, 2);
    r += __shfl_xor_sync(kFull, r, 4);
    r += __shfl_xor_sync(kFull, r, 8);
    r += __shfl_xor_sync(kFull, r, 16);
    return r;
}

// ---- geometry -------------------------------------------------------------------------------------------------
// 128 edges per block.  Wigner entries and Gaussians leave through shared memory as whole lines: a thread per edge
// storing its own 35 + 64 values would touch 32 lines per store instruction.  Memory-bound: 3.1 million edges, lmax 2, 2.0 ->
// 0.29 ms (4.8 TB/s).
template <int LMAX>
__global__ void __launch_bounds__(128)
    geometry_fwd_kernel(const float* __restrict__ pos, const int32_t* __restrict__ src, const int32_t* __restrict__ tgt,
                        const float* __restrict__ shift, const float* __restrict__ gamma, float4* __restrict__ vec,
                        float* __restrict__ env, float* __restrict__ wig, __half* __restrict__ g_hi, __half* __restrict__ g_lo,
                        BasisParams bp, int64_t num_edges) {
    pdl_sync();
    constexpr int W = Shape<LMAX>::kW;
    extern __shared__ float sm[];  // [128][W]
    __shared__ float sd[128];
    const int tid = threadIdx.x;
    const int64_t e0 = (int64_t)blockIdx.x * 128;
    const int n = (int)(num_edges - e0 < 128 ? num_edges - e0 : 128);
    if (tid < n) {
        const int64_t e = e0 + tid;
        float vx, vy, vz;
        edge_vector(pos, src, tgt, shift, e, vx, vy, vz);
        const float d = sqrtf(vx * vx + vy * vy + vz * vz);
        sd[tid] = d;
        vec[e] = make_float4(vx, vy, vz, d);
        env[e] = envelope(d, bp.cutoff);
        float q[4];
        edge_quaternion<float>(vx, vy, vz, gamma ? gamma[e] : 0.f, q);
        wigner_compact<LMAX, float>(q, [&](int i, float v) { sm[tid * W + i] = v; });
    }
    __syncthreads();
    for (int i = tid; i < n * W; i += 128) wig[e0 * W + i] = sm[i];
    const int nb = bp.num;  // multiple of 8
    for (int i = tid; i < n * (nb >> 3); i += 128) {
        const int el = i / (nb >> 3), k0 = (i % (nb >> 3)) * 8;
        uint32_t h[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float t0 = sd[el] - (bp.start + bp.step * (k0 + 2 * j)), t1 = sd[el] - (bp.start + bp.step * (k0 + 2 * j + 1));
            split_pair(expf(bp.coeff * t0 * t0), expf(bp.coeff * t1 * t1), h[j], l[j]);
        }
        const int64_t o = (e0 + el) * nb + k0;
        *reinterpret_cast<uint4*>(g_hi + o) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(g_lo + o) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

// d loss / d v per edge of a chunk from the torques, the envelope gradient and the gradient of the distance basis.
// tau_n: torque in the node frame.  tau_e: lmax 2: torque of the rotate-back in the edge frame; lmax 4: in the node
// frame; w component: envelope gradient.  Memory-bound; with the torques in place of 35 Wigner gradients an edge there is no
// Jacobian to form: 3.1 million edges 0.9 -> 0.63 ms.
template <int LMAX>
__global__ void __launch_bounds__(128)
    geometry_bwd_kernel(const float4* __restrict__ vec, const float* __restrict__ wig, const float4* __restrict__ tau_n,
                        const float4* __restrict__ tau_e, const float* __restrict__ g_gauss, float* __restrict__ grad_vec,
                        BasisParams bp, int64_t num_edges) {
    pdl_sync();
    constexpr int W = Shape<LMAX>::kW;
    __shared__ float sgd[128];
    const int tid = threadIdx.x;
    const int64_t e0 = (int64_t)blockIdx.x * 128;
    const int n = (int)(num_edges - e0 < 128 ? num_edges - e0 : 128);
    // 16 lanes per edge contract the distance-basis gradient (whole-line reads)
    for (int it = 0; it < 16; ++it) {
        const int el = it * 8 + (tid >> 4), sub = tid & 15;
        float gd = 0.f;
        if (el < n) {
            const float d = vec[e0 + el].w;
            for (int k = sub * 4; k < bp.num; k += 64) {
                const float4 g = ld4(g_gauss + (e0 + el) * bp.num + k);
                const float gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float t = d - (bp.start + bp.step * (k + j));
                    gd = fmaf(gv[j], expf(bp.coeff * t * t) * (2.0f * bp.coeff * t), gd);
                }
            }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) gd += __shfl_xor_sync(kFull, gd, o);
        if (sub == 0) sgd[el] = gd;
    }
    __syncthreads();
    if (tid >= n) return;
    const int64_t e = e0 + tid;
    const float4 v = vec[e], tn = tau_n[e], te = tau_e[e];
    float tx, ty, tz;
    if (LMAX == 2) {
        const float* r = wig + e * W + 1;  // D^1 is the Cartesian rotation
        tx = tn.x - (r[0] * te.x + r[3] * te.y + r[6] * te.z);
        ty = tn.y - (r[1] * te.x + r[4] * te.y + r[7] * te.z);
        tz = tn.z - (r[2] * te.x + r[5] * te.y + r[8] * te.z);
    } else {
        tx = tn.x + te.x;
        ty = tn.y + te.y;
        tz = tn.z + te.z;
    }
    const float d = v.w;
    const float gd = sgd[tid] + te.w * envelope_slope(d, bp.cutoff);
    const float id = d > 0.f ? 1.0f / d : 0.f, id2 = id * id, s = gd * id;
    grad_vec[e * 3 + 0] = fmaf(v.y * tz - v.z * ty, id2, s * v.x);
    grad_vec[e * 3 + 1] = fmaf(v.z * tx - v.x * tz, id2, s * v.y);
    grad_vec[e * 3 + 2] = fmaf(v.x * ty - v.y * tx, id2, s * v.z);
}

// grad_pos[n] = sign * (sum over edges leaving n - sum over edges entering n); one warp per node
__global__ void __launch_bounds__(256)
    grad_pos_kernel(const float* __restrict__ grad_vec, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ src_ptr,
                    const int32_t* __restrict__ src_perm, float* __restrict__ grad_pos, float sign, int64_t num_nodes) {
    pdl_sync();
    const int lane = threadIdx.x & 31;
    const int64_t n = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (n >= num_nodes) return;
    float x = 0.f, y = 0.f, z = 0.f;
    for (int k = src_ptr[n] + lane; k < src_ptr[n + 1]; k += 32) {
        const int64_t e = src_perm[k];
        x += grad_vec[e * 3], y += grad_vec[e * 3 + 1], z += grad_vec[e * 3 + 2];
    }
    for (int k = row_ptr[n] + lane; k < row_ptr[n + 1]; k += 32)
        x -= grad_vec[(int64_t)k * 3], y -= grad_vec[(int64_t)k * 3 + 1], z -= grad_vec[(int64_t)k * 3 + 2];
    const float t = reduce4(x, y, z, 0.f, lane);
    if (lane < 3) grad_pos[n * 3 + lane] = sign * t;
}

// copy the compact entries of one edge, times f, into this warp's shared-memory slot
template <int KW>
__device__ __forceinline__ void stage(const float* __restrict__ wig, int64_t e, float f, int lane, float* slot) {
    __syncwarp();
#pragma unroll
    for (int i = lane; i < KW; i += 32) slot[i] = wig[e * KW + i] * f;
    __syncwarp();
}

// ---- gather + rotate + radial weights -----------------------------------------------------------------------------
// out[e, row(l, m), half, :] = radial * sum_j D[(l, m), j] x[node, l^2 + j, :], node = source (half 0) or target (half 1)
template <int LMAX, int l>
__device__ __forceinline__ void gather_fwd_degrees(const float4 (&x)[Shape<LMAX>::kL], const float4 (&rad)[Shape<LMAX>::kRad],
                                                   const float* w, const OutSplit& out, int64_t o) {
    using S = Shape<LMAX>;
#pragma unroll
    for (int k = 0; k < S::rows(l); ++k) {
        const int m = k - S::mm(l);
        float4 a = f4zero();
#pragma unroll
        for (int j = 0; j < 2 * l + 1; ++j) a = fma4(w[S::woff(l) + k * (2 * l + 1) + j], x[l * l + j], a);
        out.st(o + S::mrow(l, m) * 2 * C, mul4(a, rad[S::radslot(l, m)]));
    }
    if constexpr (l < LMAX) gather_fwd_degrees<LMAX, l + 1>(x, rad, w, out, o);
}
// Bound by memory (per edge: radial weights read, planes written; node rows come from L1 and L2), so what counts is bytes
// requested ahead.  One warp per (edge, half): its node rows and radial weights, 7.5 KB (lmax 4: 18.5 KB), are all requested
// before the first is used; 20 (12) such warps fit an SM.  Halves of an edge are neighbours in a block, so that the 30 edges of
// a target find its rows in L1.  A warp per edge, a degree or a half at a time with the weights read as they are used:
// lmax 2, 129 000 edges 405 -> 380 us; lmax 4, 120 000 edges 1247 -> 799 us.  The next item's node is asked for one item ahead:
// 20 600 edges of lmax 2 72.8 -> 68.5 us, 3 240 edges of lmax 4 27.7 -> 24.3.
template <int LMAX>
__global__ void __launch_bounds__(128, LMAX == 2 ? 5 : 3)
    gather_fwd_kernel(const float* __restrict__ x, const int32_t* __restrict__ src, const int32_t* __restrict__ tgt,
                      const float* __restrict__ wig, const float* __restrict__ radial, OutSplit out, int64_t num_edges) {
    pdl_sync();
    using S = Shape<LMAX>;
    out.load_scale(nullptr);
    __shared__ float sw[4][(S::kW + 3) / 4 * 4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, c0 = lane * 4;
    float* w = sw[wid];
    auto node = [&](int64_t i) { return __ldg((i & 1 ? tgt : src) + (i >> 1)); };
    const int64_t i0 = (int64_t)blockIdx.x * 4 + wid, step = (int64_t)gridDim.x * 4;
    int next = i0 < 2 * num_edges ? node(i0) : 0;
    for (int64_t i = i0; i < 2 * num_edges; i += step) {
        const int64_t e = i >> 1;
        const int half = (int)i & 1;
        const float* x_base = x + (int64_t)next * S::kL * C + c0;
        if (i + step < 2 * num_edges) next = node(i + step);
        const float* r_base = radial + (e * S::kRad * 2 + half) * C + c0;
        float4 rad[S::kRad], xv[S::kL];
#pragma unroll
        for (int s = 0; s < S::kRad; ++s) rad[s] = ld4(r_base + s * 2 * C);
#pragma unroll
        for (int j = 0; j < S::kL; ++j) xv[j] = ld4(x_base + j * C);
        stage<S::kW>(wig, e, 1.0f, lane, w);
        gather_fwd_degrees<LMAX, 0>(xv, rad, w, out, (e * S::kM * 2 + half) * C + c0);
    }
}

// ---- rotate back + sum over the edges of a target ---------------------------------------------------------------
// MODE 0: out = residual + sum_e env W^T msg.  MODE 1 (edge-degree embedding; m = 0 rows only):
// out = [embedding of the element + system embedding on row 0] + sum / rescale.
// WPN warps share a node: each takes every WPN-th edge and the partial sums meet in shared memory.  With one warp per
// node the edges are a serial chain, which is all there is when the nodes do not fill the GPU (256 nodes, four
// layers: 0.033 ms).  Memory-bound otherwise: 129 000 edges of lmax 2 in 124 us, 5.2 TB/s (4.8 with an inverse tensor read beside).
template <int LMAX, int MODE, int WPN>
__global__ void __launch_bounds__(WPN == 1 ? 128 : 32 * WPN)
    rotate_back_kernel(const float* __restrict__ msg, const float* __restrict__ wig, const float* __restrict__ env,
                       const int32_t* __restrict__ row_ptr, int64_t e_base, const float* __restrict__ residual,
                       const float* __restrict__ emb, const int32_t* __restrict__ z, const float* __restrict__ sys,
                       const int32_t* __restrict__ batch, float* __restrict__ out, float inv_rescale, int64_t n0, int64_t n1) {
    pdl_sync();
    using S = Shape<LMAX>;
    constexpr int kWarps = WPN == 1 ? 4 : WPN;
    constexpr int rows_in = MODE == 0 ? S::kM : LMAX + 1;
    __shared__ float sw[kWarps][(S::kW + 3) / 4 * 4];
    extern __shared__ float part[];  // WPN > 1: [WPN][kL][C]
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, c0 = lane * 4;
    float* w = sw[wid];
    const int64_t stride = WPN == 1 ? (int64_t)gridDim.x * kWarps : gridDim.x;
    for (int64_t n = n0 + (WPN == 1 ? (int64_t)blockIdx.x * kWarps + wid : blockIdx.x); n < n1; n += stride) {
        const int e0 = row_ptr[n], e1 = row_ptr[n + 1];
        float4 acc[S::kL];
#pragma unroll
        for (int L = 0; L < S::kL; ++L) acc[L] = f4zero();
        for (int e = e0 + (WPN == 1 ? 0 : wid); e < e1; e += WPN) {
            const float* y_base = msg + ((int64_t)e - e_base) * rows_in * C + c0;
            float4 y[rows_in];
#pragma unroll
            for (int r = 0; r < rows_in; ++r) y[r] = ld4(y_base + r * C);
            stage<S::kW>(wig, e, env[e], lane, w);
#pragma unroll
            for (int l = 0; l <= LMAX; ++l)
#pragma unroll
                for (int k = 0; k < S::rows(l); ++k) {
                    if (MODE == 1 && k != S::mm(l)) continue;
                    const float4 yr = y[MODE == 0 ? S::mrow(l, k - S::mm(l)) : l];
#pragma unroll
                    for (int j = 0; j < 2 * l + 1; ++j)
                        acc[l * l + j] = fma4(w[S::woff(l) + k * (2 * l + 1) + j], yr, acc[l * l + j]);
                }
        }
        auto finish = [&](int L, int c, float4 v) {
            const int64_t o = (n * S::kL + L) * C + c;
            if (MODE == 1) {
                v = scale4(inv_rescale, v);
                if (L == 0) v = add4(v, add4(ld4(emb + (int64_t)z[n] * C + c), ld4(sys + (int64_t)batch[n] * C + c)));
            } else {
                v = add4(v, ld4(residual + o));
            }
            st4(out + o, v);
        };
        if (WPN == 1) {
#pragma unroll
            for (int L = 0; L < S::kL; ++L) finish(L, c0, acc[L]);
        } else {
#pragma unroll
            for (int L = 0; L < S::kL; ++L) st4(part + (wid * S::kL + L) * C + c0, acc[L]);
            __syncthreads();
            for (int L = wid; L < S::kL; L += WPN) {
                float4 v = f4zero();
#pragma unroll
                for (int i = 0; i < WPN; ++i) v = add4(v, ld4(part + (i * S::kL + L) * C + c0));
                finish(L, c0, v);
            }
            __syncthreads();
        }
    }
}

// One degree of one edge: acc = W go per row, message gradient f * acc.  lmax 2 keeps every row of W, so the torque is
// taken in the edge frame from acc and y directly; lmax 4 lacks the rows |m| > 2 there and rotates y back instead.
template <int LMAX, int MODE, int l, class Out>
__device__ __forceinline__ void rotate_back_bwd_degree(const float* __restrict__ go_base, const float* __restrict__ y_base,
                                                       const float* w, float f, const Out& grad_msg, int64_t gm, float (&t)[3],
                                                       float& ge) {
    using S = Shape<LMAX>;
    constexpr int n = 2 * l + 1, mm = S::mm(l);
    const float* wl = w + S::woff(l);
    float4 go[n];
#pragma unroll
    for (int j = 0; j < n; ++j) go[j] = ld4(go_base + (l * l + j) * C);
    auto row = [&](int k) {
        float4 a = f4zero();
#pragma unroll
        for (int j = 0; j < n; ++j) a = fma4(wl[k * n + j], go[j], a);
        return a;
    };
    if constexpr (MODE == 1) {
        const float4 y0 = ld4(y_base + l * C), a0 = row(mm);
        ge += dot4(a0, y0);
        grad_msg.st(gm + l * C, scale4(f, a0));
        if constexpr (l > 0) {
            constexpr float s0 = (float)csqrt(0.5 * l * (l + 1));
            t[0] = fmaf(s0, dot4(row(mm + 1), y0), t[0]);
            t[2] = fmaf(-s0, dot4(row(mm - 1), y0), t[2]);
        }
    } else if constexpr (LMAX == 2) {
        float4 a[n], y[n];
#pragma unroll
        for (int k = 0; k < n; ++k) y[k] = ld4(y_base + S::mrow(l, k - l) * C);
#pragma unroll
        for (int k = 0; k < n; ++k) {
            a[k] = row(k);
            ge += dot4(a[k], y[k]);
            grad_msg.st(gm + S::mrow(l, k - l) * C, scale4(f, a[k]));
        }
        torque<l>(a, y, t);
    } else {
        float4 z[n];
#pragma unroll
        for (int j = 0; j < n; ++j) z[j] = f4zero();
#pragma unroll
        for (int k = 0; k < S::rows(l); ++k) {
            const float4 y = ld4(y_base + S::mrow(l, k - mm) * C), a = row(k);
#pragma unroll
            for (int j = 0; j < n; ++j) z[j] = fma4(wl[k * n + j], y, z[j]);
            ge += dot4(a, y);
            grad_msg.st(gm + S::mrow(l, k - mm) * C, scale4(f, a));
        }
        torque<l>(z, go, t);
    }
}

// backward of the same, one warp per edge: gradient of the message rows (half planes for MODE 0, float32 for MODE 1),
// torque and envelope gradient, stored or added to tau_e.  Memory-bound (gradient rows of a target come from L1 and L2): 129 000
// edges of lmax 2 in 242 us, 7.5 TB/s of requested bytes, against 4.8 with 35 Wigner gradients to reduce; grid of whole waves.
template <int LMAX, int MODE, class Out>
__global__ void __launch_bounds__(128, LMAX == 2 ? 4 : 3)
    rotate_back_bwd_kernel(const float* __restrict__ grad_out, const float* __restrict__ msg, const float* __restrict__ wig,
                           const float* __restrict__ env, const int32_t* __restrict__ tgt, Out grad_msg,
                           const float* __restrict__ scale_ptr, float* __restrict__ tau_e, int accumulate, float inv_rescale,
                           int64_t e_base, int64_t num_edges) {
    pdl_sync();
    using S = Shape<LMAX>;
    grad_msg.load_scale(scale_ptr);
    constexpr int rows_in = MODE == 0 ? S::kM : LMAX + 1;
    __shared__ float sw[4][(S::kW + 3) / 4 * 4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, c0 = lane * 4;
    float* w = sw[wid];
    for (int64_t i = (int64_t)blockIdx.x * 4 + wid; i < num_edges; i += (int64_t)gridDim.x * 4) {
        const int64_t e = e_base + i;
        stage<S::kW>(wig, e, 1.0f, lane, w);
        const float* go_base = grad_out + (int64_t)tgt[e] * S::kL * C + c0;
        const float* y_base = msg + i * rows_in * C + c0;
        const int64_t gm = i * rows_in * C + c0;
        const float f = env[e] * inv_rescale;
        float t[3] = {0.f, 0.f, 0.f}, ge = 0.f;
        rotate_back_bwd_degree<LMAX, MODE, 0>(go_base, y_base, w, f, grad_msg, gm, t, ge);
        rotate_back_bwd_degree<LMAX, MODE, 1>(go_base, y_base, w, f, grad_msg, gm, t, ge);
        rotate_back_bwd_degree<LMAX, MODE, 2>(go_base, y_base, w, f, grad_msg, gm, t, ge);
        if constexpr (LMAX == 4) {
            rotate_back_bwd_degree<LMAX, MODE, 3>(go_base, y_base, w, f, grad_msg, gm, t, ge);
            rotate_back_bwd_degree<LMAX, MODE, 4>(go_base, y_base, w, f, grad_msg, gm, t, ge);
        }
        if constexpr (LMAX == 4 && MODE == 1) {  // the m = 0 rows give the torque in the edge frame: turn it
            const float a = t[0], b = t[1], c = t[2];
            t[0] = -(w[1] * a + w[4] * b + w[7] * c);
            t[1] = -(w[2] * a + w[5] * b + w[8] * c);
            t[2] = -(w[3] * a + w[6] * b + w[9] * c);
        }
        const float r = reduce4(t[0] * f, t[1] * f, t[2] * f, ge * inv_rescale, lane);
        if (lane < 4) tau_e[e * 4 + lane] = accumulate ? tau_e[e * 4 + lane] + r : r;
    }
}

// ---- gather + rotate + radial scale, backward, summed per node ----------------------------------------------------
// One edge, degrees l..LHI: node gradient, radial gradient and torque from the gradient rows of the rotated edge (go) and
// the radial weights (rd), both in the order of the pass: rows (l, m = -mm..mm), slots (l, |m|).
template <int LMAX, int l, int LLO, int LHI, int NR, int NS, int R, int S0, class RadOut>
__device__ __forceinline__ void gather_bwd_degrees(const float4 (&go)[NR], const float4 (&rd)[NS], const RadOut& grad_radial,
                                                   int64_t rad_base, const float* w,
                                                   const float4 (&xv)[(LHI + 1) * (LHI + 1) - LLO * LLO],
                                                   float4 (&acc)[(LHI + 1) * (LHI + 1) - LLO * LLO], float (&t)[3]) {
    using S = Shape<LMAX>;
    constexpr int n = 2 * l + 1, mm = S::mm(l), X = l * l - LLO * LLO;
    const float* wl = w + S::woff(l) - S::woff(LLO);
    float4 x[n], g[n];
#pragma unroll
    for (int j = 0; j < n; ++j) {
        x[j] = xv[X + j];
        g[j] = f4zero();
    }
#pragma unroll
    for (int am = 0; am <= mm; ++am) {
        float4 dr = f4zero();
#pragma unroll
        for (int sgn = 0; sgn < (am ? 2 : 1); ++sgn) {
            const int k = mm + (sgn ? -am : am);
            float4 rot = f4zero();
#pragma unroll
            for (int j = 0; j < n; ++j) rot = fma4(wl[k * n + j], x[j], rot);
            dr = add4(dr, mul4(go[R + k], rot));
            const float4 gr = mul4(go[R + k], rd[S0 + am]);
#pragma unroll
            for (int j = 0; j < n; ++j) g[j] = fma4(wl[k * n + j], gr, g[j]);
        }
        grad_radial.st(rad_base + S::radslot(l, am) * 2 * C, dr);
    }
#pragma unroll
    for (int j = 0; j < n; ++j) acc[X + j] = add4(acc[X + j], g[j]);
    torque<l>(g, x, t);
    if constexpr (l < LHI)
        gather_bwd_degrees<LMAX, l + 1, LLO, LHI, NR, NS, R + 2 * mm + 1, S0 + mm + 1>(go, rd, grad_radial, rad_base, w, xv, acc, t);
}

template <int LMAX> __host__ __device__ constexpr int rows_of(int lo, int hi) {
    int s = 0;
    for (int l = lo; l <= hi; ++l) s += Shape<LMAX>::rows(l);
    return s;
}
template <int LMAX> __host__ __device__ constexpr int slots_of(int lo, int hi) {
    int s = 0;
    for (int l = lo; l <= hi; ++l) s += Shape<LMAX>::mm(l) + 1;
    return s;
}

__device__ __forceinline__ void copy_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// lmax 4, by source: a chunk holds few edges of a source, and its three passes would each begin with an empty stage
template <int LMAX, int HALF> constexpr bool ahead = LMAX == 2 || HALF == 1;
constexpr int kGatherRows = 15;  // rows and radial weights of an edge in the widest pass (degrees 0-2)

// HALF 0: source columns, the node's edges through perm (by-source order); HALF 1: target columns, consecutive edges.
// Degrees LLO..LHI in one pass over the node's edges.  Bound by memory once enough of it is asked for at a time: a warp
// walks its edges in turn.  The gradient rows and radial weights of the next edge are copied to shared memory (two stages
// of 7.5 KB a warp, every lane the 16 bytes of a row that it reads itself, so nothing has to synchronise) while this one
// is worked on.  us per launch, all rows of an edge requested when its turn came -> this: 129 000 edges of lmax 2, by source
// 344 -> 307, by target 299 -> 250; 120 000 edges of lmax 4, by target 834 -> 660, by source 805 -> 890, hence ahead<>.
template <int LMAX, int LLO, int LHI, int HALF, int STEP, class RadOut>
__device__ __forceinline__ void gather_bwd_pass(const float* __restrict__ grad, const float* __restrict__ x_base,
                                                const float* __restrict__ wig, const float* __restrict__ radial,
                                                const RadOut& grad_radial, const int32_t* __restrict__ perm,
                                                float* __restrict__ tau, bool add_tau, int64_t e_base, int eb, int ee, int lane,
                                                float* w, float* stages, float4 (&acc)[(LHI + 1) * (LHI + 1) - LLO * LLO]) {
    using S = Shape<LMAX>;
    constexpr int kRows = (LHI + 1) * (LHI + 1) - LLO * LLO, R0 = LLO * LLO;
    constexpr int W0 = S::woff(LLO), WN = S::woff(LHI + 1) - W0;
    constexpr int NR = rows_of<LMAX>(LLO, LHI), NS = slots_of<LMAX>(LLO, LHI);
    static_assert(WN <= 64, "two Wigner entries a lane");
    static_assert(NR + NS <= kGatherRows, "a stage");
    constexpr bool kAhead = ahead<LMAX, HALF>;
    const int c0 = lane * 4;
    float4 xv[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        xv[r] = ld4(x_base + (R0 + r) * C + c0);
        acc[r] = f4zero();
    }
    if (eb >= ee) return;
    auto edge = [&](int k) -> int64_t { return HALF == 0 ? (int64_t)__ldg(perm + k) : (int64_t)k; };
    // every gradient row (l, m) and radial weight (l, |m|) of edge row i of the chunk's buffers, in the order of the pass
    auto rows = [&](int64_t i, auto&& use) {
        const float* go = grad + i * (int64_t)S::kM * 2 * C + HALF * C + c0;
        const float* rd = radial + i * (int64_t)S::kRad * 2 * C + HALF * C + c0;
        int r = 0;
#pragma unroll
        for (int l = LLO; l <= LHI; ++l) {
#pragma unroll
            for (int m = -S::mm(l); m <= S::mm(l); ++m) use(r++, go + S::mrow(l, m) * 2 * C);
        }
#pragma unroll
        for (int l = LLO; l <= LHI; ++l) {
#pragma unroll
            for (int am = 0; am <= S::mm(l); ++am) use(r++, rd + S::radslot(l, am) * 2 * C);
        }
    };
    auto request = [&](int64_t i, int stage) {
        float* dst = stages + stage * kGatherRows * C + c0;
        if constexpr (kAhead) rows(i, [&](int r, const float* p) { copy_async16(dst + r * C, p); });
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    int64_t e = edge(eb), next = eb + STEP < ee ? edge(eb + STEP) : 0;  // global edges
    request(e - e_base, 0);
    commit();
    float w0 = lane < WN ? __ldg(wig + e * S::kW + W0 + lane) : 0.f, w1 = lane + 32 < WN ? __ldg(wig + e * S::kW + W0 + 32 + lane) : 0.f;
    int stage = 0;
    for (int k = eb; k < ee; k += STEP, stage ^= 1) {
        const int64_t ecur = e;
        float4 v[NR + NS];
        if constexpr (!kAhead) rows(e - e_base, [&](int r, const float* p) { v[r] = __ldcs(reinterpret_cast<const float4*>(p)); });
        const int64_t rad_base = (e - e_base) * (int64_t)S::kRad * 2 * C + HALF * C + c0;
        const bool more = k + STEP < ee;
        if (more) {
            e = next;
            request(e - e_base, stage ^ 1);
            if (k + 2 * STEP < ee) next = edge(k + 2 * STEP);
        }
        commit();
        float told = 0.f;
        if (add_tau && lane < 3) told = tau[ecur * 4 + lane];
        __syncwarp();
        if (lane < WN) w[lane] = w0;
        if (lane + 32 < WN) w[lane + 32] = w1;
        __syncwarp();
        if (more) {
            w0 = lane < WN ? __ldg(wig + e * S::kW + W0 + lane) : 0.f;
            w1 = lane + 32 < WN ? __ldg(wig + e * S::kW + W0 + 32 + lane) : 0.f;
        }
        if constexpr (kAhead) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
#pragma unroll
            for (int r = 0; r < NR + NS; ++r) v[r] = ld4(stages + (stage * kGatherRows + r) * C + c0);
        }
        float4 go[NR], rd[NS];
#pragma unroll
        for (int r = 0; r < NR; ++r) go[r] = v[r];
#pragma unroll
        for (int r = 0; r < NS; ++r) rd[r] = v[NR + r];
        float t[3] = {0.f, 0.f, 0.f};
        gather_bwd_degrees<LMAX, LLO, LLO, LHI, NR, NS, 0, 0>(go, rd, grad_radial, rad_base, w, xv, acc, t);
        const float r = reduce4(t[0], t[1], t[2], 0.f, lane);
        if (lane < 3) tau[ecur * 4 + lane] = told + r;
    }
}

template <int LMAX, int HALF, int WPN, class RadOut>
__global__ void __launch_bounds__(WPN == 1 ? 128 : 32 * WPN, WPN == 8 ? 1 : 3)
    gather_bwd_kernel(const float* __restrict__ grad, const float* __restrict__ x, const int32_t* __restrict__ lo,
                      const int32_t* __restrict__ hi, const int32_t* __restrict__ perm, const float* __restrict__ wig,
                      const float* __restrict__ radial, float* __restrict__ gx, int store_gx, float* __restrict__ tau, int store_tau,
                      RadOut grad_radial, const float* __restrict__ scale_ptr, int64_t e_base, int64_t n0, int64_t n1) {
    pdl_sync();
    using S = Shape<LMAX>;
    grad_radial.load_scale(scale_ptr);
    constexpr int kWarps = WPN == 1 ? 4 : WPN;
    __shared__ float sw[kWarps][48];
    extern __shared__ float4 gather_stages[];  // a warp's two stages; WPN > 1: then its partial sums
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, c0 = lane * 4;
    constexpr int kMine = 2 * kGatherRows * C;
    float* stages = reinterpret_cast<float*>(gather_stages) + wid * kMine;
    const int64_t stride = WPN == 1 ? (int64_t)gridDim.x * kWarps : gridDim.x;
    for (int64_t n = n0 + (WPN == 1 ? (int64_t)blockIdx.x * kWarps + wid : blockIdx.x); n < n1; n += stride) {
        const int eb = lo[n], ee = hi[n];
        if (eb == ee && !store_gx) continue;  // store_gx: the first contribution to every node's gradient
        const float* x_base = x + n * (int64_t)S::kL * C;
        float* g_base = gx + n * (int64_t)S::kL * C;
        auto pass = [&](auto lo_tag, auto hi_tag, bool add_tau) {
            constexpr int LLO = decltype(lo_tag)::value, LHI = decltype(hi_tag)::value;
            constexpr int kRows = (LHI + 1) * (LHI + 1) - LLO * LLO;
            float4 acc[kRows];
            gather_bwd_pass<LMAX, LLO, LHI, HALF, WPN>(grad, x_base, wig, radial, grad_radial, perm, tau, add_tau, e_base,
                                                       eb + (WPN == 1 ? 0 : wid), ee, lane, sw[wid], stages, acc);
            if (WPN == 1) {
#pragma unroll
                for (int r = 0; r < kRows; ++r) {
                    float* o = g_base + (LLO * LLO + r) * C + c0;
                    st4(o, store_gx ? acc[r] : add4(ld4(o), acc[r]));
                }
            } else {
#pragma unroll
                for (int r = 0; r < kRows; ++r) st4(stages + r * C + c0, acc[r]);
                __syncthreads();
                for (int r = wid; r < kRows; r += WPN) {
                    float* o = g_base + (LLO * LLO + r) * C + c0;
                    float4 v = store_gx ? f4zero() : ld4(o);
#pragma unroll
                    for (int i = 0; i < WPN; ++i) v = add4(v, ld4(stages + (i - wid) * kMine + r * C + c0));
                    st4(o, v);
                }
                __syncthreads();
            }
        };
        using std::integral_constant;
        pass(integral_constant<int, 0>{}, integral_constant<int, 2>{}, !store_tau);
        if constexpr (LMAX == 4) {
            pass(integral_constant<int, 3>{}, integral_constant<int, 3>{}, true);
            pass(integral_constant<int, 4>{}, integral_constant<int, 4>{}, true);
        }
    }
}

}  // namespace step
}  // namespace fcb200
