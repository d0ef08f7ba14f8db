// Radius graph and index tables of one evaluation with a single host read (the edge count), for fcb200_model_*.
//
// The stand-alone path (radius_graph.cu behind graph.py) reads bounds, candidate total and edge total back and builds
// its CSR and by-source tables from library sorts: 6 host reads and ~100 launches, 2-20 ms of host time with an idle
// GPU.  Here one kernel per evaluation finds the candidates of a target and applies the neighbour limit while they sit
// in shared memory, a scan turns the counts into the CSR (and the chunk boundaries), and four short kernels write the
// edges and the by-source order.  The arithmetic that decides membership is radius_graph.cuh's, so the edge set is the
// same bit for bit.
#include "radius_graph.cuh"

namespace fcb200 {
namespace step {

constexpr int kCap = 512;        // candidates of one target held in shared memory
constexpr int kMaxChunks = 512;  // chunk boundaries in the info block
enum { kInfoEdges = 0, kInfoFlag = 1, kInfoChunks = 2, kInfoMoved = 3, kInfoSources = 4, kInfoCells = 5, kInfoPairs = 6, kInfoInput = 7, kInfoNodes = 8,
       kInfoEdgeCut = 8 + kMaxChunks + 1 };
static_assert(FCB200_GRAPH_INFO_WORDS >= 8 + 2 * (kMaxChunks + 1), "info block");

__device__ __forceinline__ float cross_rn(float a, float b, float c, float d) { return __fsub_rn(__fmul_rn(a, b), __fmul_rn(c, d)); }
__device__ __forceinline__ float sum3_rn(float a, float b, float c) { return __fadd_rn(__fadd_rn(a, b), c); }

// periodic images along one lattice vector: ceil(r |a_j x a_k| / |V|) in float32
__device__ int image_repeats(const float* cr, float vol, float radius, int* __restrict__ flag) {
    const float x = __fdiv_rn(cr[0], vol), y = __fdiv_rn(cr[1], vol), z = __fdiv_rn(cr[2], vol);
    const float inv = __fsqrt_rn(sum3_rn(__fmul_rn(x, x), __fmul_rn(y, y), __fmul_rn(z, z)));
    const float r = ceilf(__fmul_rn(radius, inv));
    if (!(r <= 100.f)) {  // degenerate cell: left to the general path
        *flag = 1;
        return 0;
    }
    return (int)r;
}

// what of the inputs lies outside the embedding tables, the host's to report: a sweep of all blocks over the atoms
__device__ __forceinline__ void check_inputs(const int64_t* __restrict__ z64, const int64_t* __restrict__ batch64, int64_t num_nodes,
                                             int num_elements, const int64_t* __restrict__ charge, const int64_t* __restrict__ spin,
                                             int nsys, int32_t* __restrict__ info) {
    int bits = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < num_nodes; i += (int64_t)gridDim.x * blockDim.x) {
        if (z64[i] < 0 || z64[i] >= num_elements) bits |= FCB200_INPUT_ELEMENT;
        if (batch64[i] < 0 || batch64[i] >= nsys) bits |= FCB200_INPUT_BATCH;
    }
    if (threadIdx.x == 0) {
        if (charge && (charge[blockIdx.x] < -100 || charge[blockIdx.x] > 100)) bits |= FCB200_INPUT_CHARGE;
        if (spin && (spin[blockIdx.x] < 0 || spin[blockIdx.x] > 100)) bits |= FCB200_INPUT_SPIN;
    }
    if (bits) atomicOr(info + kInfoInput, bits);
}

// One block per system: atom range, bounding box, image counts -> system table.  Grid cells as build_system_table sizes
// them (edge radius / 1.99, coarser when the product of the dimensions would exceed the limit).
__global__ void __launch_bounds__(1024)
    graph_systems_kernel(int64_t num_nodes, const float* __restrict__ pos, const float* __restrict__ cell, const uint8_t* __restrict__ pbc,
                         const int64_t* __restrict__ natoms, int nsys, float radius, const int64_t* __restrict__ z64,
                         const int64_t* __restrict__ batch64, int num_elements, const int64_t* __restrict__ charge,
                         const int64_t* __restrict__ spin, int32_t* __restrict__ sys, float* __restrict__ bbox, int32_t* __restrict__ info) {
    pdl_sync();
    check_inputs(z64, batch64, num_nodes, num_elements, charge, spin, nsys, info);
    __shared__ long long s_begin[32];
    __shared__ float s_lo[32][3], s_hi[32][3];
    const int s = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, threads = blockDim.x, warps = threads >> 5;
    long long before = 0;
    for (int i = tid; i < s; i += threads) before += natoms[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(kFull, before, o);
    if (lane == 0) s_begin[wid] = before;
    __syncthreads();
    before = 0;
    for (int i = 0; i < warps; ++i) before += s_begin[i];
    // counts that do not add up to the positions given are the general path's to report
    const bool bad = before + natoms[s] > num_nodes || natoms[s] < 0;
    const int a0 = bad ? 0 : (int)before, a1 = bad ? 0 : a0 + (int)natoms[s];
    if (bad && tid == 0) info[kInfoFlag] = 1;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int a = a0 + tid; a < a1; a += threads)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float v = pos[(int64_t)a * 3 + k];
            lo[k] = fminf(lo[k], v), hi[k] = fmaxf(hi[k], v);
        }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(kFull, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(kFull, hi[k], o));
        }
        if (lane == 0) s_lo[wid][k] = lo[k], s_hi[wid][k] = hi[k];
    }
    __syncthreads();
    if (tid != 0) return;
    for (int w = 1; w < warps; ++w)
        for (int k = 0; k < 3; ++k) lo[k] = fminf(lo[k], s_lo[w][k]), hi[k] = fmaxf(hi[k], s_hi[w][k]);
    const float* c = cell + (int64_t)s * 9;
    const float c23[3] = {cross_rn(c[4], c[8], c[5], c[7]), cross_rn(c[5], c[6], c[3], c[8]), cross_rn(c[3], c[7], c[4], c[6])};
    const float c31[3] = {cross_rn(c[7], c[2], c[8], c[1]), cross_rn(c[8], c[0], c[6], c[2]), cross_rn(c[6], c[1], c[7], c[0])};
    const float c12[3] = {cross_rn(c[1], c[5], c[2], c[4]), cross_rn(c[2], c[3], c[0], c[5]), cross_rn(c[0], c[4], c[1], c[3])};
    const float vol = sum3_rn(__fmul_rn(c[0], c23[0]), __fmul_rn(c[1], c23[1]), __fmul_rn(c[2], c23[2]));
    int32_t* w = sys + (int64_t)s * FCB200_SYS_WORDS;
    int rep[3];
    rep[0] = pbc[s * 3 + 0] ? image_repeats(c23, vol, radius, info + kInfoFlag) : 0;
    rep[1] = pbc[s * 3 + 1] ? image_repeats(c31, vol, radius, info + kInfoFlag) : 0;
    rep[2] = pbc[s * 3 + 2] ? image_repeats(c12, vol, radius, info + kInfoFlag) : 0;
    w[0] = a0, w[1] = a1;
    w[2] = rep[0], w[3] = rep[1], w[4] = rep[2];
    w[5] = (2 * rep[0] + 1) * (2 * rep[1] + 1) * (2 * rep[2] + 1);
    float h = radius / 1.99f;
    float dim[3];
    const float limit = (float)((1 << 24) / nsys);
    for (;;) {
        for (int k = 0; k < 3; ++k) dim[k] = floorf((hi[k] - lo[k] + 2.f * (radius + 1e-3f)) / h) + 1.f;
        if (a1 <= a0) dim[0] = dim[1] = dim[2] = 1.f;
        if (!(dim[0] * dim[1] * dim[2] > limit) || h > 1e30f) break;
        h *= 1.26f;
    }
    for (int k = 0; k < 3; ++k) {
        w[8 + k] = (int)dim[k];
        w[11 + k] = __float_as_int(lo[k] - radius - 1e-3f);
        bbox[s * 6 + k] = lo[k];
        bbox[s * 6 + 3 + k] = hi[k];
    }
    w[14] = __float_as_int(1.0f / h);
    for (int i = 0; i < 9; ++i) w[15 + i] = __float_as_int(c[i]);
}

// first source and first grid cell of every system, and their totals; one warp, latency-bound (1 system 3 us, 257: 45)
__global__ void __launch_bounds__(32) graph_offsets_kernel(int32_t* __restrict__ sys, int nsys, int32_t* __restrict__ info) {
    pdl_sync();
    if (threadIdx.x != 0) return;
    long long src = 0, cells = 0;
    double pairs = 0.0;
    for (int s = 0; s < nsys; ++s) {
        int32_t* w = sys + (int64_t)s * FCB200_SYS_WORDS;
        const long long n = w[1] - w[0];
        w[6] = (int)src, w[7] = (int)cells;
        src += n * w[5];
        cells += (long long)w[8] * w[9] * w[10];
        pairs += (double)n * (double)n * w[5];
    }
    if (src >= (1LL << 31) || cells >= (1LL << 31)) info[kInfoFlag] = 1;
    info[kInfoSources] = (int)src, info[kInfoCells] = (int)cells;
    info[kInfoPairs] = __float_as_int((float)pairs);
}

__global__ void graph_convert_kernel(const int64_t* __restrict__ z64, const int64_t* __restrict__ batch64, int32_t* __restrict__ z,
                                     int32_t* __restrict__ batch, int64_t n, int num_elements, int nsys, int32_t* __restrict__ info) {
    pdl_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 8) info[i] = 0;  // the kernels that raise words of it run after this one
    if (i >= n) return;
    const int64_t a = z64[i], b = batch64[i];
    const bool bad = a < 0 || a >= num_elements || b < 0 || b >= nsys;  // reported by the next kernel
    z[i] = bad ? 0 : (int)a;
    batch[i] = bad ? 0 : (int)b;
}

// Has a kept candidate list expired?  Any atom that moved by more than the limit, or another cell, split or periodicity.
__global__ void graph_moved_kernel(const float* __restrict__ pos, const float* __restrict__ pos0, float limit_sq, int64_t n,
                                   const float* __restrict__ cell, const float* __restrict__ cell0, const uint8_t* __restrict__ pbc,
                                   const uint8_t* __restrict__ pbc0, const int64_t* __restrict__ natoms, const int64_t* __restrict__ natoms0,
                                   int nsys, int32_t* __restrict__ info) {
    pdl_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool moved = false;
    if (i < n) {
        const float dx = pos[i * 3] - pos0[i * 3], dy = pos[i * 3 + 1] - pos0[i * 3 + 1], dz = pos[i * 3 + 2] - pos0[i * 3 + 2];
        moved = !(dx * dx + dy * dy + dz * dz <= limit_sq);
    }
    if (i < nsys * 9LL) moved = moved || cell[i] != cell0[i];
    if (i < nsys * 3LL) moved = moved || (pbc[i] != 0) != (pbc0[i] != 0);
    if (i < nsys) moved = moved || natoms[i] != natoms0[i];
    if (moved) info[kInfoMoved] = 1;
}

// One warp per target: candidates within the radius into shared memory (MODE 0: every periodic image whose bounding box
// is in reach, atom by atom; 1: grid cells; 2: a kept list, at the current positions), then the max-neighbour rule of
// rg_select_kernel, then the kept ones (source atom, packed image) to the target's row of `rows`.  Bound by instruction issue
// and shared memory: 25 000 atoms 0.17 ms, 256 atoms 0.022.
template <int MODE>
__global__ void __launch_bounds__(256)
    graph_select_kernel(const float* __restrict__ pos, const int32_t* __restrict__ sys, int nsys, const int32_t* __restrict__ batch,
                        const float* __restrict__ bbox, const int32_t* __restrict__ cell_ptr, const float4* __restrict__ bucket,
                        const int32_t* __restrict__ cand_ptr, const int32_t* __restrict__ cand_id, float radius, float radius_sq,
                        int max_neighbors, int2* __restrict__ rows, int stride, int32_t* __restrict__ count, int32_t* __restrict__ info,
                        int64_t num_nodes) {
    pdl_sync();
    __shared__ float s_d2[8][kCap];
    __shared__ int2 s_id[8][kCap];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t t = (int64_t)blockIdx.x * 8 + wid;
    if (t >= num_nodes) return;
    float* d2s = s_d2[wid];
    int2* ids = s_id[wid];
    const Sys s = load_sys(sys, batch[t]);
    const float tx = pos[t * 3 + 0], ty = pos[t * 3 + 1], tz = pos[t * 3 + 2];
    int m = 0;
    auto add = [&](bool keep, float d2, int atom, int code) {
        const unsigned mask = __ballot_sync(kFull, keep);
        const int at = m + __popc(mask & ((1u << lane) - 1u));
        if (keep && at < kCap) d2s[at] = d2, ids[at] = make_int2(atom, code);
        m += __popc(mask);
    };
    auto code_of = [](int n0, int n1, int n2) { return (n0 + 128) | ((n1 + 128) << 8) | ((n2 + 128) << 16); };
    if (MODE == 0) {
        const float* bb = bbox + batch[t] * 6;
        const float reach = radius_sq * 1.001f + 1e-2f;  // rounding of the box test never drops an image
        for (int img = 0; img < s.nimg; ++img) {
            int n0, n1, n2;
            decode_image(s, img, n0, n1, n2);
            const float zero[3] = {0.f, 0.f, 0.f};
            float ox, oy, oz;
            image_position(s, zero, 0, n0, n1, n2, ox, oy, oz);
            const float bx = fmaxf(fmaxf(bb[0] + ox - tx, tx - (bb[3] + ox)), 0.f), by = fmaxf(fmaxf(bb[1] + oy - ty, ty - (bb[4] + oy)), 0.f),
                        bz = fmaxf(fmaxf(bb[2] + oz - tz, tz - (bb[5] + oz)), 0.f);
            if (bx * bx + by * by + bz * bz > reach) continue;
            for (int a = s.atom_begin; a < s.atom_end; a += 32) {
                const int i = a + lane;
                float d2 = 0.f;
                if (i < s.atom_end) {
                    float px, py, pz;
                    image_position(s, pos, i, n0, n1, n2, px, py, pz);
                    d2 = dist_sq(tx, ty, tz, make_float4(px, py, pz, 0.f));
                }
                add(d2 <= radius_sq && d2 != 0.f, d2, i, code_of(n0, n1, n2));
            }
        }
    } else if (MODE == 1) {
        int gx, gy, gz;
        grid_coords(s, tx, ty, tz, gx, gy, gz);
        gx = min(max(gx, 0), s.d0 - 1), gy = min(max(gy, 0), s.d1 - 1), gz = min(max(gz, 0), s.d2 - 1);
        int b = 0, e = 0;
        if (lane < 25) {
            const int yy = gy + lane / 5 - 2, zz = gz + lane % 5 - 2;
            if (yy >= 0 && yy < s.d1 && zz >= 0 && zz < s.d2) {
                const int x0 = max(gx - 2, 0), x1 = min(gx + 2, s.d0 - 1);
                const int c0 = s.grid_begin + x0 + s.d0 * (yy + s.d1 * zz);
                b = cell_ptr[c0], e = cell_ptr[c0 + (x1 - x0) + 1];
            }
        }
        for (int row = 0; row < 25; ++row) {
            const int rb = __shfl_sync(kFull, b, row), re = __shfl_sync(kFull, e, row);
            for (int i0 = rb; i0 < re; i0 += 32) {
                const int i = i0 + lane;
                float d2 = 0.f;
                int sid = s.source_begin;
                if (i < re) {
                    const float4 sp = bucket[i];
                    d2 = dist_sq(tx, ty, tz, sp);
                    sid = __float_as_int(sp.w);
                }
                const int local = sid - s.source_begin;
                int n0, n1, n2;
                decode_image(s, local % s.nimg, n0, n1, n2);
                add(d2 <= radius_sq && d2 != 0.f, d2, s.atom_begin + local / s.nimg, code_of(n0, n1, n2));
            }
        }
    } else {
        const int b = cand_ptr[t], e = cand_ptr[t + 1];
        for (int i0 = b; i0 < e; i0 += 32) {
            const int i = i0 + lane;
            float d2 = 0.f;
            int atom = 0, code = 0;
            const int local = i < e ? cand_id[i] - s.source_begin : -1;
            // an expired list, whose result the host discards, may name sources that this system does not have
            if (local >= 0 && local < (s.atom_end - s.atom_begin) * s.nimg) {
                int n0, n1, n2;
                decode_image(s, local % s.nimg, n0, n1, n2);
                atom = s.atom_begin + local / s.nimg;
                float px, py, pz;
                image_position(s, pos, atom, n0, n1, n2, px, py, pz);
                d2 = dist_sq(tx, ty, tz, make_float4(px, py, pz, 0.f));
                code = code_of(n0, n1, n2);
            }
            add(d2 <= radius_sq && d2 != 0.f, d2, atom, code);
        }
    }
    if (m > kCap) {
        if (lane == 0) info[kInfoFlag] = 1;
        m = kCap;
    }
    __syncwarp();
    constexpr unsigned kInf = 0x7f800000u;
    float thr = __uint_as_float(kInf - 1u);
    if (max_neighbors > 0 && m > max_neighbors) {
        unsigned lo = 0u, hi = __float_as_uint(radius_sq);
        while (lo < hi) {
            const unsigned mid = lo + ((hi - lo) >> 1);
            int c = 0;
            for (int i = lane; i < m; i += 32) c += (__float_as_uint(d2s[i]) <= mid) ? 1 : 0;
            c = warp_sum_i(c);
            if (c >= max_neighbors + 1) hi = mid; else lo = mid + 1;
        }
        thr = fminf(__fadd_rn(__uint_as_float(lo), 0.01f), thr);
    }
    int kept = 0;
    for (int i0 = 0; i0 < m; i0 += 32) {
        const int i = i0 + lane;
        const bool keep = i < m && d2s[i] <= thr;
        const unsigned mask = __ballot_sync(kFull, keep);
        const int at = kept + __popc(mask & ((1u << lane) - 1u));
        if (keep && at < stride) rows[t * stride + at] = ids[i];
        kept += __popc(mask);
    }
    if (lane == 0) {
        if (kept > stride) info[kInfoFlag] = 1;
        count[t] = min(kept, stride);
    }
}

// exclusive scan by one block (latency-bound; 25 000 counts 24 us, 256: 3 us); with info: the total and the chunk boundaries (node whose first edge reaches c * E / chunks)
__global__ void __launch_bounds__(1024)
    graph_scan_kernel(const int32_t* __restrict__ counts, int32_t* __restrict__ ptr, int64_t n, int chunk_edges, int32_t* __restrict__ info) {
    pdl_sync();
    __shared__ int warp_tot[32];
    __shared__ int carry;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int64_t base = 0; base < n; base += 8192) {
        const int64_t i0 = base + (int64_t)tid * 8;
        int v[8], tsum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) tsum += v[j] = i0 + j < n ? counts[i0 + j] : 0;
        int incl = tsum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) warp_tot[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            const int t0 = warp_tot[lane];
            int wi = t0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(kFull, wi, o);
                if (lane >= o) wi += u;
            }
            warp_tot[lane] = wi - t0;
        }
        __syncthreads();
        int run = carry + warp_tot[wid] + incl - tsum;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (i0 + j < n) ptr[i0 + j] = run;
            run += v[j];
        }
        __syncthreads();
        if (tid == 1023) carry = run;
        __syncthreads();
    }
    const int total = carry;
    if (tid == 0) ptr[n] = total;
    if (info == nullptr) return;
    __syncthreads();
    const int chunks = max(1, min(kMaxChunks, (int)(((int64_t)total + chunk_edges / 2) / chunk_edges)));
    for (int c = tid; c <= chunks; c += 1024) {
        int node = c == 0 ? 0 : (int)n;
        if (c > 0 && c < chunks) {
            const int want = (int)((int64_t)total * c / chunks);
            int lo = 0, hi = (int)n;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (ptr[mid] < want) lo = mid + 1; else hi = mid;
            }
            node = lo;
        }
        info[kInfoNodes + c] = node;
        info[kInfoEdgeCut + c] = c == chunks ? total : ptr[node];
    }
    if (tid == 0) {
        info[kInfoEdges] = total;
        info[kInfoChunks] = chunks;
    }
}

// rows -> edge arrays (int32 for the kernels, the reference's int64 edge_index and float offsets), shift vectors, and the
// number of edges leaving each node
__global__ void __launch_bounds__(256)
    graph_fill_kernel(const int32_t* __restrict__ sys, const int32_t* __restrict__ batch, const int2* __restrict__ rows, int stride,
                      const int32_t* __restrict__ row_ptr, int32_t* __restrict__ src, int32_t* __restrict__ tgt, float* __restrict__ shift,
                      int64_t* __restrict__ edge_index, float* __restrict__ offsets, int32_t* __restrict__ src_count, int64_t num_edges,
                      int64_t num_nodes) {
    pdl_sync();
    const int lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (t >= num_nodes) return;
    const int b = row_ptr[t], m = row_ptr[t + 1] - b;
    const float* c = reinterpret_cast<const float*>(sys + (int64_t)batch[t] * FCB200_SYS_WORDS + 15);
    for (int i = lane; i < m; i += 32) {
        const int2 r = rows[t * stride + i];
        const int64_t e = b + i;
        const float n0 = (float)((r.y & 255) - 128), n1 = (float)(((r.y >> 8) & 255) - 128), n2 = (float)(((r.y >> 16) & 255) - 128);
        src[e] = r.x;
        tgt[e] = (int)t;
        edge_index[e] = r.x;
        edge_index[num_edges + e] = t;
        offsets[e * 3 + 0] = n0, offsets[e * 3 + 1] = n1, offsets[e * 3 + 2] = n2;
#pragma unroll
        for (int k = 0; k < 3; ++k) shift[e * 3 + k] = n0 * c[k] + n1 * c[3 + k] + n2 * c[6 + k];
        if (src_count) atomicAdd(src_count + r.x, 1);
    }
}

__global__ void graph_count_kernel(const int32_t* __restrict__ node, int32_t* __restrict__ count, int64_t num_edges) {
    pdl_sync();
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < num_edges) atomicAdd(count + node[e], 1);
}

// edges into their source's segment, in any order ...
__global__ void graph_bucket_kernel(const int32_t* __restrict__ src, const int32_t* __restrict__ src_ptr, int32_t* __restrict__ left,
                                    int32_t* __restrict__ unsorted, const int32_t* __restrict__ num_edges) {
    pdl_sync();
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= *num_edges) return;  // the arrays may be larger than the edge list
    const int s = src[e];
    unsorted[src_ptr[s] + atomicSub(left + s, 1) - 1] = (int)e;
}
// ... and each segment (a few dozen edges) in edge order, by counting the smaller ids.  Also, per chunk, the first
// position of the segment whose edge belongs to that chunk or a later one.
__global__ void __launch_bounds__(256)
    graph_order_kernel(const int32_t* __restrict__ unsorted, const int32_t* __restrict__ src_ptr, int32_t* __restrict__ perm,
                       int32_t* __restrict__ chunk_src, const int32_t* __restrict__ edge_cut, int chunks, int64_t num_nodes) {
    pdl_sync();
    const int lane = threadIdx.x & 31;
    const int64_t n = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (n >= num_nodes) return;
    const int b = src_ptr[n], e = src_ptr[n + 1];
    for (int i = b + lane; i < e; i += 32) {
        const int v = unsorted[i];
        int rank = 0;
        for (int j = b; j < e; ++j) rank += unsorted[j] < v ? 1 : 0;
        perm[b + rank] = v;
    }
    if (chunk_src == nullptr) return;
    for (int c = lane; c <= chunks; c += 32) {
        const int cut = edge_cut[c];
        int below = 0;
        for (int j = b; j < e; ++j) below += unsorted[j] < cut ? 1 : 0;
        chunk_src[(int64_t)c * num_nodes + n] = b + below;
    }
}

// short kernels of a small graph: see launch_pdl
struct PdlScope {
    explicit PdlScope(int64_t nodes) { pdl_launches = nodes * 30 <= kPdlEdges; }
    ~PdlScope() { pdl_launches = false; }
};

}  // namespace step
}  // namespace fcb200

using namespace fcb200;

extern "C" {

int fcb200_graph_systems(const fcb200_graph* g, void* stream) {
    if (!g || g->num_nodes < 1 || g->num_systems < 1 || !(g->radius > 0.f)) return FCB200_EINVAL;
    if (!g->pos || !g->cell || !g->pbc || !g->natoms || !g->batch64 || !g->z64 || !g->sys || !g->bbox || !g->z || !g->batch || !g->info)
        return FCB200_EINVAL;
    const step::PdlScope scope(g->num_nodes);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    launch_pdl(step::graph_convert_kernel, dim3((unsigned)((g->num_nodes + 255) / 256)), dim3(256), 0, st, g->z64, g->batch64, g->z, g->batch, g->num_nodes,
                                                                                      g->num_elements, g->num_systems, g->info);
    // few systems: a block each has to sweep many atoms
    launch_pdl(step::graph_systems_kernel, dim3(g->num_systems), dim3(g->num_systems < 148 ? 1024 : 128), 0, st, g->num_nodes, g->pos, g->cell, g->pbc, g->natoms, g->num_systems, g->radius, g->z64,
                                                               g->batch64, g->num_elements, g->charge, g->spin, g->sys, g->bbox, g->info);
    if (g->want_totals) launch_pdl(step::graph_offsets_kernel, dim3(1), dim3(32), 0, st, g->sys, g->num_systems, g->info);
    return launch_status();
}

int fcb200_graph_select(const fcb200_graph* g, void* stream) {
    if (!g || g->num_nodes < 1 || !g->rows || !g->count || !g->row_ptr || g->stride < 1 || g->chunk_edges < 1) return FCB200_EINVAL;
    const step::PdlScope scope(g->num_nodes);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned grid = (unsigned)((g->num_nodes + 7) / 8);
    const float r2 = g->radius_sq;
    if (g->cand_ptr) {
        if (!g->cand_id || !g->cand_sys) return FCB200_EINVAL;
        if (g->pos0) {
            if (!g->cell0 || !g->pbc0 || !g->natoms0) return FCB200_EINVAL;
            const int64_t n = g->num_nodes > 9LL * g->num_systems ? g->num_nodes : 9LL * g->num_systems;
            launch_pdl(step::graph_moved_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, g->pos, g->pos0, g->limit_sq, g->num_nodes, g->cell, g->cell0,
                                                                                  g->pbc, g->pbc0, g->natoms, g->natoms0, g->num_systems, g->info);
        }
        launch_pdl(step::graph_select_kernel<2>, dim3(grid), dim3(256), 0, st, g->pos, g->cand_sys, g->num_systems, g->batch, nullptr, nullptr, nullptr, g->cand_ptr,
                                                           g->cand_id, g->radius, r2, g->max_neighbors, reinterpret_cast<int2*>(g->rows),
                                                           g->stride, g->count, g->info, g->num_nodes);
    } else if (g->cell_ptr) {
        if (!g->cell_count || !g->source_cell || !g->cell_fill || !g->bucket || g->num_cells < 1) return FCB200_EINVAL;
        if (cudaMemsetAsync(g->cell_count, 0, (size_t)(g->num_cells + 1) * 4, st) != cudaSuccess) return launch_status();
        if (cudaMemsetAsync(g->cell_fill, 0, (size_t)(g->num_cells + 1) * 4, st) != cudaSuccess) return launch_status();
        int rc = fcb200_rg_count_sources(g->pos, g->sys, g->num_systems, g->num_sources, g->cell_count, g->source_cell, stream);
        if (rc) return rc;
        launch_pdl(step::graph_scan_kernel, dim3(1), dim3(1024), 0, st, g->cell_count, g->cell_ptr, g->num_cells, 1, nullptr);
        rc = fcb200_rg_fill_buckets(g->pos, g->sys, g->num_systems, g->num_sources, g->source_cell, g->cell_ptr, g->cell_fill, g->bucket,
                                    g->num_cells, stream);
        if (rc) return rc;
        launch_pdl(step::graph_select_kernel<1>, dim3(grid), dim3(256), 0, st, g->pos, g->sys, g->num_systems, g->batch, nullptr, g->cell_ptr,
                                                           reinterpret_cast<const float4*>(g->bucket), nullptr, nullptr, g->radius, r2,
                                                           g->max_neighbors, reinterpret_cast<int2*>(g->rows), g->stride, g->count, g->info,
                                                           g->num_nodes);
    } else {
        launch_pdl(step::graph_select_kernel<0>, dim3(grid), dim3(256), 0, st, g->pos, g->sys, g->num_systems, g->batch, g->bbox, nullptr, nullptr, nullptr, nullptr,
                                                           g->radius, r2, g->max_neighbors, reinterpret_cast<int2*>(g->rows), g->stride, g->count,
                                                           g->info, g->num_nodes);
    }
    launch_pdl(step::graph_scan_kernel, dim3(1), dim3(1024), 0, st, g->count, g->row_ptr, g->num_nodes, g->chunk_edges, g->info);
    return launch_status();
}

int fcb200_graph_fill(const fcb200_graph* g, void* stream) {
    if (!g || g->num_edges < 1 || !g->src || !g->tgt || !g->row_ptr) return FCB200_EINVAL;
    const step::PdlScope scope(g->num_nodes);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t n = g->num_nodes, e = g->num_edges;
    const unsigned gn = (unsigned)((n + 7) / 8), ge = (unsigned)((e + 255) / 256);
    if (g->src_ptr) {
        if (!g->src_count || !g->src_tmp || !g->src_perm) return FCB200_EINVAL;
        if (cudaMemsetAsync(g->src_count, 0, (size_t)n * 4, st) != cudaSuccess) return launch_status();
    }
    if (g->rows) {
        if (!g->shift || !g->edge_index || !g->cell_offsets || !g->batch) return FCB200_EINVAL;
        launch_pdl(step::graph_fill_kernel, dim3(gn), dim3(256), 0, st, g->cand_sys ? g->cand_sys : g->sys, g->batch, reinterpret_cast<const int2*>(g->rows), g->stride,
                                                    g->row_ptr, g->src, g->tgt, g->shift, g->edge_index, g->cell_offsets,
                                                    g->src_ptr ? g->src_count : nullptr, e, n);
    } else {  // edges given by the caller, sorted by target: row_ptr and the by-source counts from them
        if (!g->count) return FCB200_EINVAL;
        if (cudaMemsetAsync(g->count, 0, (size_t)n * 4, st) != cudaSuccess) return launch_status();
        launch_pdl(step::graph_count_kernel, dim3(ge), dim3(256), 0, st, g->tgt, g->count, e);
        launch_pdl(step::graph_scan_kernel, dim3(1), dim3(1024), 0, st, g->count, g->row_ptr, n, g->chunk_edges, g->info);
        if (g->src_ptr) launch_pdl(step::graph_count_kernel, dim3(ge), dim3(256), 0, st, g->src, g->src_count, e);
    }
    if (g->src_ptr) {
        launch_pdl(step::graph_scan_kernel, dim3(1), dim3(1024), 0, st, g->src_count, g->src_ptr, n, 1, nullptr);
        launch_pdl(step::graph_bucket_kernel, dim3(ge), dim3(256), 0, st, g->src, g->src_ptr, g->src_count, g->src_tmp, g->row_ptr + n);
        launch_pdl(step::graph_order_kernel, dim3(gn), dim3(256), 0, st, g->src_tmp, g->src_ptr, g->src_perm, g->chunk_src, g->info + step::kInfoEdgeCut,
                                                     g->num_chunks, n);
    }
    return launch_status();
}

}  // extern "C"
