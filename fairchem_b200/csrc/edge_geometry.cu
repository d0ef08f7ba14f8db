// Per-edge geometry: edge vector, length, envelope, Gaussian basis and the compact Wigner-D of the
// rotation that takes the edge direction to +Y (l <= 2, or l <= 4 with rows |m| <= 2), forward and backward.
//
// The rotation code is written once as a template over the scalar type.  Instantiated with
// float it is the forward pass; instantiated with Dual3 (value + three tangents, one per component
// of the edge vector) it yields d(wigner)/d(vec) exactly, which the backward kernel contracts with
// the incoming gradient.  35 outputs against 3 inputs makes forward mode the cheap direction.
#include "geometry.cuh"

namespace fcb200 {

template <int LMAX>
__global__ void __launch_bounds__(128)
    edge_geometry_fwd_kernel(const float* __restrict__ pos, const int32_t* __restrict__ src, const int32_t* __restrict__ tgt,
                             const float* __restrict__ shift, const float* __restrict__ gamma, float* __restrict__ vec,
                             float* __restrict__ dist, float* __restrict__ env, float* __restrict__ wig,
                             float* __restrict__ gauss, BasisParams bp, int64_t num_edges) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= num_edges) return;
    float vx, vy, vz;
    edge_vector(pos, src, tgt, shift, e, vx, vy, vz);
    const float d = sqrtf(vx * vx + vy * vy + vz * vz);
    if (vec) { vec[e * 3 + 0] = vx; vec[e * 3 + 1] = vy; vec[e * 3 + 2] = vz; }
    if (dist) dist[e] = d;
    if (env) env[e] = envelope(d, bp.cutoff);
    if (gauss) {
        for (int k = 0; k < bp.num; ++k) {
            const float t = d - (bp.start + bp.step * k);
            gauss[e * bp.num + k] = expf(bp.coeff * t * t);
        }
    }
    if (wig) {
        float q[4];
        edge_quaternion<float>(vx, vy, vz, gamma ? gamma[e] : 0.f, q);
        float* w = wig + e * Shape<LMAX>::kW;
        wigner_compact<LMAX, float>(q, [&](int i, float v) { w[i] = v; });
    }
}

template <int LMAX>
__global__ void __launch_bounds__(128)
    edge_geometry_bwd_kernel(const float* __restrict__ pos, const int32_t* __restrict__ src, const int32_t* __restrict__ tgt,
                             const float* __restrict__ shift, const float* __restrict__ gamma,
                             const float* __restrict__ grad_wig, const float* __restrict__ grad_env,
                             const float* __restrict__ grad_gauss, const float* __restrict__ grad_dist,
                             float* __restrict__ grad_vec, BasisParams bp, int64_t num_edges) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= num_edges) return;
    float vx, vy, vz;
    edge_vector(pos, src, tgt, shift, e, vx, vy, vz);
    const float d = sqrtf(vx * vx + vy * vy + vz * vz);
    float gx = 0.f, gy = 0.f, gz = 0.f;
    // scalar chain through the length
    float gd = grad_dist ? grad_dist[e] : 0.f;
    if (grad_env) gd += grad_env[e] * envelope_slope(d, bp.cutoff);
    if (grad_gauss) {
        for (int k = 0; k < bp.num; ++k) {
            const float t = d - (bp.start + bp.step * k);
            gd += grad_gauss[e * bp.num + k] * expf(bp.coeff * t * t) * (2.0f * bp.coeff * t);
        }
    }
    if (d > 0.f) {
        const float s = gd / d;
        gx = s * vx; gy = s * vy; gz = s * vz;
    }
    if (grad_wig) {
        Dual3 q[4];
        const Dual3 dx{vx, 1.f, 0.f, 0.f}, dy{vy, 0.f, 1.f, 0.f}, dz{vz, 0.f, 0.f, 1.f};
        edge_quaternion<Dual3>(dx, dy, dz, gamma ? gamma[e] : 0.f, q);
        const float* gw = grad_wig + e * Shape<LMAX>::kW;
        wigner_compact<LMAX, Dual3>(q, [&](int i, Dual3 v) {
            const float g = gw[i];
            gx = fmaf(g, v.a, gx);
            gy = fmaf(g, v.b, gy);
            gz = fmaf(g, v.c, gz);
        });
    }
    grad_vec[e * 3 + 0] = gx;
    grad_vec[e * 3 + 1] = gy;
    grad_vec[e * 3 + 2] = gz;
}

}  // namespace fcb200

using namespace fcb200;

extern "C" {

int fcb200_lx_edge_geometry_fwd(const float* pos, const int32_t* src, const int32_t* tgt, const float* shift, const float* gamma,
                                float* vec, float* dist, float* env, float* wig, float* gauss, float cutoff, int32_t num_basis,
                                float basis_start, float basis_stop, float basis_width, int64_t num_edges, int64_t num_nodes,
                                int32_t lmax, void* stream) {
    if (!pos || !src || !tgt || num_edges < 0 || num_nodes < 0 || cutoff <= 0.f) return FCB200_EINVAL;
    if (gauss && num_basis < 2) return FCB200_EINVAL;
    if (lmax != 2 && lmax != 4) return FCB200_EINVAL;
    if (num_edges == 0) return FCB200_OK;
    const BasisParams bp = make_basis(cutoff, num_basis, basis_start, basis_stop, basis_width);
    const unsigned grid = (unsigned)((num_edges + 127) / 128);
    if (lmax == 2)
        edge_geometry_fwd_kernel<2><<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(pos, src, tgt, shift, gamma, vec, dist, env,
                                                                                         wig, gauss, bp, num_edges);
    else
        edge_geometry_fwd_kernel<4><<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(pos, src, tgt, shift, gamma, vec, dist, env,
                                                                                         wig, gauss, bp, num_edges);
    return launch_status();
}

int fcb200_lx_edge_geometry_bwd(const float* pos, const int32_t* src, const int32_t* tgt, const float* shift, const float* gamma,
                                const float* grad_wig, const float* grad_env, const float* grad_gauss, const float* grad_dist,
                                float* grad_vec, float cutoff, int32_t num_basis, float basis_start, float basis_stop,
                                float basis_width, int64_t num_edges, int64_t num_nodes, int32_t lmax, void* stream) {
    if (!pos || !src || !tgt || !grad_vec || num_edges < 0 || num_nodes < 0 || cutoff <= 0.f) return FCB200_EINVAL;
    if (grad_gauss && num_basis < 2) return FCB200_EINVAL;
    if (lmax != 2 && lmax != 4) return FCB200_EINVAL;
    if (num_edges == 0) return FCB200_OK;
    const BasisParams bp = make_basis(cutoff, num_basis, basis_start, basis_stop, basis_width);
    const unsigned grid = (unsigned)((num_edges + 127) / 128);
    if (lmax == 2)
        edge_geometry_bwd_kernel<2><<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
            pos, src, tgt, shift, gamma, grad_wig, grad_env, grad_gauss, grad_dist, grad_vec, bp, num_edges);
    else
        edge_geometry_bwd_kernel<4><<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
            pos, src, tgt, shift, gamma, grad_wig, grad_env, grad_gauss, grad_dist, grad_vec, bp, num_edges);
    return launch_status();
}

int fcb200_edge_geometry_fwd(const float* pos, const int32_t* src, const int32_t* tgt, const float* shift, const float* gamma,
                             float* vec, float* dist, float* env, float* wig, float* gauss, float cutoff, int32_t num_basis,
                             float basis_start, float basis_stop, float basis_width, int64_t num_edges, int64_t num_nodes,
                             void* stream) {
    return fcb200_lx_edge_geometry_fwd(pos, src, tgt, shift, gamma, vec, dist, env, wig, gauss, cutoff, num_basis, basis_start,
                                       basis_stop, basis_width, num_edges, num_nodes, 2, stream);
}

int fcb200_edge_geometry_bwd(const float* pos, const int32_t* src, const int32_t* tgt, const float* shift, const float* gamma,
                             const float* grad_wig, const float* grad_env, const float* grad_gauss, const float* grad_dist,
                             float* grad_vec, float cutoff, int32_t num_basis, float basis_start, float basis_stop,
                             float basis_width, int64_t num_edges, int64_t num_nodes, void* stream) {
    return fcb200_lx_edge_geometry_bwd(pos, src, tgt, shift, gamma, grad_wig, grad_env, grad_gauss, grad_dist, grad_vec, cutoff,
                                       num_basis, basis_start, basis_stop, basis_width, num_edges, num_nodes, 2, stream);
}

}  // extern "C"
