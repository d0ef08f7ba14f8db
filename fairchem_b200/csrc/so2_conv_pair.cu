// The SO(2) convolution launches of so2_conv_fused.cu on CTA pairs (tcgen05 cta_group::2), for launches with enough rows:
// plain tile lists and the forward gate.
//
// Two CTAs of a cluster own 256 rows and walk output tiles of 256 columns (two listed 128-column tiles that read the same
// input columns; a tile without a partner is 128 wide).  One thread of the leader issues M = 256 MMAs that read each CTA's
// own rows and half of the weight rows from each CTA, so per 64-deep k-step a CTA takes 64 KiB from L2 and moves 160 KiB
// through its shared-memory port for 1536 cycles of MMA, where the single form takes 128 KiB and moves 288 KiB.
// All 512 columns of tensor memory hold one tile's main and correction accumulators.  The epilogue therefore empties them
// into registers first (a thread's 128 sums; the first 32 wait in shared memory) and hands them back before it works on
// them; the tensor core waits some 3300 cycles a tile for that, of 18 000 it works on one of the first convolution.  (The
// main sums handed back ahead of the corrections, so that one half is emptied while the other is worked on: the reads then
// share tensor memory with the products and take as much longer, 1118 -> 1166 thousand cycles a launch.)
// Epilogue: lane = row, 32 columns at a time, for every tile of the list, so gates stay in registers; a 32 x 32 block leaves
// through the warp's 4 KiB of shared memory as a TMA store (whole lines, rows past the end are clipped).
//
// What bounds it at size is the power cap: back to back launches of either form run at 985 W (a us is a mJ), so what counts is
// energy, and half the operand traffic is what this form saves.  us a launch, alone / on pairs, one board: first convolution, lmax 2,
// 131 072 rows 1040 / 980; lmax 4, 60 000 rows 1796 / 1594; second convolution, lmax 2, 131 072 rows 435 / 410; first convolution's
// backward 940 / 872.  (The forward kind spills 128 bytes a thread, the plain one 40.)
#include "so2_conv.cuh"

namespace fcb200 {
namespace fused {
namespace pair {

constexpr int kStages = 3;
constexpr int kStageBytes = 4 * kPart;               // A_hi | A_lo | W_hi | W_lo: 128 rows each, of W at most
constexpr int kEpiWarps = 8;
constexpr int kThreads = 128 + 32 * kEpiWarps;       // warp 0 TMA, warp 1 MMA (leader), 2-3 idle, warps 4-11 epilogue
constexpr int kIdleRegs = 40, kEpiRegs = 232;
static_assert(128 * kIdleRegs + 32 * kEpiWarps * kEpiRegs <= kThreads * 168, "register split");
constexpr int kTmemCols = 512, kCorr = 256;          // main sums in columns [0, 256), corrections in [256, 512)
constexpr int kSmemBytes = kStages * kStageBytes + kEpiWarps * 4096 + 1024 + 256;
static_assert(8 * (2 * kStages + 2) + 12 <= 256, "barrier block");

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Load into this CTA's shared memory whose bytes are counted on a barrier that may be the peer's.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar), "l"(policy)
        : "memory");
}
// arrive on the barrier at this offset in both CTAs once the MMAs issued so far are complete
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}
// M = 256 (128 rows in each CTA), N columns, half of whose operand rows are in each CTA
template <int N>
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
    constexpr uint32_t desc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8, %9, %10, %11, %12}, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(desc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}

struct Maps {
    CUtensorMap a[2], w[6];  // hi, lo; boxes of 128 (A) and 64 (W) rows by 64 columns
    CUtensorMap y, o[2];     // 32 x 32 blocks of y and of the output planes
};

template <int KIND>
__device__ __forceinline__ void epilogue(const Maps& maps, const PairPlan& plan, const Params& prm, int row_off, uint32_t tmem_base,
                                         uint32_t tile, uint32_t tfull, uint32_t tempty, volatile int* abort_flag, volatile int* range_flag) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = warp & 3, half = (warp - 4) >> 2;
    const float a_scale = prm.a_scale ? *prm.a_scale : 1.0f;
    const float o_scale = prm.o_scale ? *prm.o_scale : 1.0f;
    const uint64_t policy = l2_policy_evict_first();
    __half2 top = __floats2half2_rn(0.f, 0.f);
    f32x2 keepv[KIND == kPlainKind ? 1 : 2][16];  // o_scale * sigmoid of the degree's gate, per chunk
    const uint32_t own = tile + (uint32_t)(lane * 128);  // the lane's row of a float32 block, 16-byte units swizzled
    auto put = [](uint32_t at, f32x2 a, f32x2 b) { asm volatile("st.shared.v2.b64 [%0], {%1,%2};" ::"r"(at), "l"(a), "l"(b) : "memory"); };
    auto get = [](uint32_t at, f32x2& a, f32x2& b) { asm volatile("ld.shared.v2.b64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "r"(at) : "memory"); };
    // the block that left last has been read from shared memory
    auto tile_free = [&] {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
    };
    uint32_t phase = 0;
    int64_t mt;
    int g;
    for (int64_t n = 0; plan.order.item(n, gridDim.x >> 1, blockIdx.x >> 1, mt, g); ++n) {
        const int64_t row0 = mt * 2 * BM + row_off + q * 32;
        const bool live = row0 < prm.m_total;
        auto store = [&](const CUtensorMap* map, uint32_t from, int col) { tma_store_2d_hint(map, from, col, (int)row0, policy); };
        auto commit = [] { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); };
        auto emit_y = [&](const f32x2 (&x)[16], int col) {
            tile_free();
#pragma unroll
            for (int v = 0; v < 8; ++v) put(own + (uint32_t)((v ^ (lane & 7)) * 16), x[2 * v], x[2 * v + 1]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0 && live) {
                store(&maps.y, tile, col);
                commit();
            }
        };
        auto emit_planes = [&](const f32x2 (&x)[16], int col) {
            uint32_t h[16], l[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) split2(x[i], h[i], l[i], top);
            tile_free();
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t at = tile + (uint32_t)(lane * 64 + ((u ^ ((lane >> 1) & 3)) * 16));
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(h[4 * u]), "r"(h[4 * u + 1]), "r"(h[4 * u + 2]), "r"(h[4 * u + 3]) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at + 2048u), "r"(l[4 * u]), "r"(l[4 * u + 1]), "r"(l[4 * u + 2]), "r"(l[4 * u + 3]) : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0 && live) {
                store(&maps.o[0], tile, col);
                store(&maps.o[1], tile + 2048u, col);
                commit();
            }
        };
        for (int ti = plan.begin[g]; ti < plan.begin[g + 1]; ++ti, phase ^= 1) {
            const PairTile& t = plan.t[ti];
            bool ok = mbar_wait(tfull, phase, abort_flag);
            ok = __all_sync(kFull, ok);
            if (!ok) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem_base + (uint32_t)(half * 64) + ((uint32_t)(q * 32) << 16);
            f32x2 poison = 0;  // becomes NaN if any value is inf or NaN (an overflowed half upstream)
            f32x2 v[4][16];    // [0] waits in shared memory while the others are fetched
            auto take = [&](int j) {
                uint32_t r[32], c[32];
                const uint32_t from = acc + (uint32_t)((j >> 1) * BN + (j & 1) * 32);
                FCB_TMEM_LD32(r, from);
                FCB_TMEM_LD32(c, from + kCorr);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const f32x2 lo = pack(1.0f / kLoScale, 1.0f / kLoScale);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    v[j][i] = fma2(pack(__uint_as_float(c[2 * i]), __uint_as_float(c[2 * i + 1])), lo, pack(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
                    poison = fma2(v[j][i], 0, poison);
                }
            };
            take(0);
            tile_free();
#pragma unroll
            for (int i = 0; i < 8; ++i) put(own + (uint32_t)((i ^ (lane & 7)) * 16), v[0][2 * i], v[0][2 * i + 1]);
            take(1);
            if (t.n > 1) {
                take(2);
                take(3);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(tempty);
#pragma unroll
            for (int i = 0; i < 8; ++i) get(own + (uint32_t)((i ^ (lane & 7)) * 16), v[0][2 * i], v[0][2 * i + 1]);
            {
                float p0, p1;
                unpack(poison, p0, p1);
                if (!(p0 + p1 == 0.f)) *range_flag = 1;
            }
            const float out_scale = 1.0f / (a_scale * prm.w_scale[t.w]);  // a power of two: scaling after the sum is exact
            const f32x2 os2 = pack(out_scale, out_scale);
#pragma unroll 1
            for (int s = 0; s < t.n; ++s) {
                const int mode = t.mode[s], flags = t.flags[s];
                const float* bias = prm.bias[t.w] ? prm.bias[t.w] + t.w_row[s] + half * 64 : nullptr;
#pragma unroll
                for (int c2 = 0; c2 < 2; ++c2) {
                    const int col = half * 64 + c2 * 32;
                    f32x2(&x)[16] = v[c2];
                    if (bias) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 b = ld4(bias + c2 * 32 + 4 * i);
                            x[2 * i] = fma2(x[2 * i], os2, pack(b.x, b.y)), x[2 * i + 1] = fma2(x[2 * i + 1], os2, pack(b.z, b.w));
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) x[i] = fma2(x[i], os2, 0);
                    }
                    if (KIND == kPlainKind || mode == kPlain) {
                        emit_y(x, t.out_col[s] + col);
                        if constexpr (KIND == kForwardKind) {
                            if (flags & kGateSrc) {
                                const bool twice = (flags & kGateSilu) != 0;
                                auto gate_of = [&](float g) { return o_scale * sigmoid_f(twice ? g * sigmoid_f(g) : g); };
#pragma unroll
                                for (int i = 0; i < 16; ++i) keepv[c2][i] = map2(x[i], gate_of);
                            }
                        }
                    } else if constexpr (KIND == kForwardKind) {
                        if (flags & kKeep) emit_y(x, t.y_col[s] + col);
                        if (mode == kSilu) {
                            auto sig = [&](float g) { return o_scale * sigmoid_f(g); };
#pragma unroll
                            for (int i = 0; i < 16; ++i) x[i] = mul2(x[i], map2(x[i], sig));
                        } else {
#pragma unroll
                            for (int i = 0; i < 16; ++i) x[i] = mul2(x[i], keepv[c2][i]);
                        }
                        emit_planes(x, t.out_col[s] + col);
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) v[0][i] = v[2][i], v[1][i] = v[3][i];
            }
        }
    }
    if (!(__half2float(__hmax_nan(__low2half(top), __high2half(top))) <= kHalfMax)) *range_flag = 1;  // inf or NaN
}

// All products of one tile, issued by one lane of a warp that walks the loop as one (see so2_conv_fused.cu).  s, ph: ring stage that comes next and its parity.
template <int N>
__device__ __forceinline__ bool tile_products(uint64_t desc0, uint32_t tmem, int k, uint32_t full0, uint32_t empty0, int& s, uint32_t& ph, volatile int* abort_flag) {
    constexpr uint64_t kLo = kPart >> 4, kW = 2 * (kPart >> 4), kStep = 2;  // in a stage, 16-byte units
    const int num_kb = (k + KB - 1) / KB, tail = (k - (num_kb - 1) * KB + 15) / 16;  // columns past k belong to a neighbour
    for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(full0 + 8u * s, ph, abort_flag)) return false;  // both CTAs' operands have landed
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t d = desc0 + (uint64_t)(s * (kStageBytes >> 4));
        const int steps = kb + 1 == num_kb ? tail : KB / 16;
        if (elect_one()) {
#pragma unroll
            for (int j = 0; j < KB / 16; ++j) {
                if (j >= steps) break;
                const uint32_t add = kb > 0 || j > 0;
                umma_f16_pair<N>(tmem, d + j * kStep, d + kW + j * kStep, add);
                umma_f16_pair<N>(tmem + kCorr, d + j * kStep, d + kW + kLo + j * kStep, add);
                umma_f16_pair<N>(tmem + kCorr, d + kLo + j * kStep, d + kW + j * kStep, 1u);
            }
            umma_commit_pair(empty0 + 8u * s);
        }
        __syncwarp();
        if (++s == kStages) s = 0, ph ^= 1;
    }
    return true;
}

template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    so2_conv_pair_kernel(const __grid_constant__ Maps maps, const __grid_constant__ PairPlan plan, const __grid_constant__ Params prm) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t epi_base = base + kStages * kStageBytes;
    const uint32_t bar_base = epi_base + kEpiWarps * 4096;
    // barrier block: full[S] | empty[S] | tmem full | tmem empty | tmem slot, abort flag, range flag.  full[] and tmem empty
    // are used in the leader only.
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
    const uint32_t tfull = bar_base + 8u * (2 * kStages), tempty = tfull + 8u;
    uint8_t* const bar_generic = smem_raw + (bar_base - smem_u32(smem_raw));
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_generic + 8 * (2 * kStages + 2));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_generic + 8 * (2 * kStages + 2) + 4);
    volatile int* range_flag = reinterpret_cast<volatile int*>(bar_generic + 8 * (2 * kStages + 2) + 8);
    auto part_addr = [&](int s, int which) { return base + s * kStageBytes + which * kPart; };

    const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar(s), 1);   // the leader announces both CTAs' bytes
            mbar_init(empty_bar(s), 1);  // the leader's commit, delivered to both CTAs
        }
        mbar_init(tfull, 1);
        mbar_init(tempty, 2 * kEpiWarps);  // one lane of every epilogue warp of both CTAs
        *abort_flag = 0;
        *range_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)),
                     "r"((uint32_t)kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (warp == 2 && lane < 11) prefetch_map(lane < 2 ? &maps.a[lane] : lane < 8 ? &maps.w[lane - 2] : lane == 8 ? &maps.y : &maps.o[lane - 9]);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers are initialised before either signals the other
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    pdl_sync();  // barriers and tensor memory are set up while the predecessor finishes

    if (warp >= 4) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpiRegs));
        epilogue<KIND>(maps, plan, prm, (int)rank * BM, tmem_base, epi_base + (uint32_t)((warp - 4) * 4096), tfull, map_to_cta(tempty, 0), abort_flag, range_flag);
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIdleRegs));
        if (warp == 0 && lane == 0) {
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            // an A tile is fetched again for each of the output tiles of its m-block, the weights by every pair: keep
            // both in L2 ahead of the streamed outputs
            const uint64_t keep = l2_policy_evict_last();
            int64_t mt;
            int g;
            for (int64_t n = 0; ok && plan.order.item(n, gridDim.x >> 1, blockIdx.x >> 1, mt, g); ++n) {
                const int row = (int)(mt * 2 * BM + rank * BM);
                for (int ti = plan.begin[g]; ti < plan.begin[g + 1] && ok; ++ti) {
                    const PairTile& t = plan.t[ti];
                    const CUtensorMap *whi = &maps.w[2 * t.w], *wlo = &maps.w[2 * t.w + 1];
                    const bool wide = t.n > 1;
                    const int w_row = wide ? t.w_row[rank] : t.w_row[0] + 64 * (int)rank;  // this CTA's half of the tile's columns
                    const int num_kb = (t.k + KB - 1) / KB;
                    for (int kb = 0; kb < num_kb; ++kb) {
                        ok = mbar_wait(empty_bar(s), ph, abort_flag);
                        if (!ok) break;
                        const uint32_t bar = map_to_cta(full_bar(s), 0);
                        if (leader) mbar_expect_tx(full_bar(s), 2u * (wide ? 4 * kPart : 3 * kPart));
                        tma_load_2d_pair(part_addr(s, 0), &maps.a[0], t.a_col + kb * KB, row, bar, keep);
                        tma_load_2d_pair(part_addr(s, 2), whi, kb * KB, w_row, bar, keep);
                        if (wide) tma_load_2d_pair(part_addr(s, 2) + kPart / 2, whi, kb * KB, w_row + 64, bar, keep);
                        tma_load_2d_pair(part_addr(s, 3), wlo, kb * KB, w_row, bar, keep);
                        if (wide) tma_load_2d_pair(part_addr(s, 3) + kPart / 2, wlo, kb * KB, w_row + 64, bar, keep);
                        tma_load_2d_pair(part_addr(s, 1), &maps.a[1], t.a_col + kb * KB, row, bar, keep);
                        if (++s == kStages) s = 0, ph ^= 1;
                    }
                }
            }
        }
        if (warp == 1 && leader) {
            int s = 0;
            uint32_t ph = 0, acc_free = 1;
            bool ok = true;
            const uint64_t desc0 = smem_desc128(base);
            int64_t mt;
            int g;
            for (int64_t n = 0; ok && plan.order.item(n, gridDim.x >> 1, blockIdx.x >> 1, mt, g); ++n) {
                for (int ti = plan.begin[g]; ti < plan.begin[g + 1] && ok; ++ti, acc_free ^= 1) {
                    ok = mbar_wait_warp(tempty, acc_free, abort_flag);  // both epilogues have emptied the accumulators
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const int k = plan.t[ti].k;
                    if (plan.t[ti].n > 1) ok = tile_products<2 * BN>(desc0, tmem_base, k, full_bar(0), empty_bar(0), s, ph, abort_flag);
                    else ok = tile_products<BN>(desc0, tmem_base, k, full_bar(0), empty_bar(0), s, ph, abort_flag);
                    if (ok && elect_one()) umma_commit_pair(tfull);
                    __syncwarp();
                }
            }
        }
    }

    settle(abort_flag);
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves, nor frees tensor memory, while its peer can still reach it
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
    }
    if (threadIdx.x == 0 && prm.status) {
        if (*abort_flag) atomicExch(prm.status, 1);
        else if (*range_flag) atomicCAS(prm.status, 0, 2);
    }
}

static int map_2d(CUtensorMap* map, CUtensorMapDataType type, int size, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_cols, int box_rows,
                  CUtensorMapSwizzle swizzle) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return FCB200_EINVAL;
    cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t gstride[1] = {(cuuint64_t)ld * size};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, type, 2, const_cast<void*>(ptr), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? FCB200_OK : FCB200_EINVAL;
}
static int map_half(CUtensorMap* map, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
    return map_2d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, ptr, rows, cols, ld, KB, box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace pair

int launch_pair(const PairPlan& plan, const Params& prm, const void* a_hi, const void* a_lo, int64_t lda, int64_t a_cols, const void* const* w_hi,
                const void* const* w_lo, const int64_t* w_rows, const int64_t* w_cols, const bool (&used)[3], int64_t o_cols, bool forward, cudaStream_t st) {
    using namespace pair;
    Maps maps;
    const int64_t m = prm.m_total;
    int rc = map_half(&maps.a[0], a_hi, m, a_cols, lda, BM);
    if (!rc) rc = map_half(&maps.a[1], a_lo, m, a_cols, lda, BM);
    int first = -1;
    for (int i = 0; i < 3 && !rc; ++i) {
        if (!used[i]) continue;
        if (first < 0) first = i;
        rc = map_half(&maps.w[2 * i], w_hi[i], w_rows[i], w_cols[i], w_cols[i], 64);
        if (!rc) rc = map_half(&maps.w[2 * i + 1], w_lo[i], w_rows[i], w_cols[i], w_cols[i], 64);
    }
    // a list without float32 tiles need not have a column of y, one without split tiles no planes: those have no map
    const bool stores_y = prm.y_cols > 0;
    if (!rc && stores_y) rc = map_2d(&maps.y, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, prm.y, m, prm.y_cols, prm.ldy, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!rc && forward) {
        rc = map_2d(&maps.o[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, prm.o_hi, m, o_cols, prm.ldo, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
        if (!rc) rc = map_2d(&maps.o[1], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, prm.o_lo, m, o_cols, prm.ldo, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
    }
    if (!stores_y) maps.y = maps.o[0];
    if (!forward) maps.o[0] = maps.o[1] = maps.y;
    if (rc) return rc;
    for (int i = 0; i < 3; ++i)
        if (!used[i]) maps.w[2 * i] = maps.w[2 * first], maps.w[2 * i + 1] = maps.w[2 * first + 1];
    const int64_t items = plan.order.rows * plan.order.groups;
    const int64_t pairs = sm_count() / 2;
    const int grid = 2 * (int)(items < pairs ? items : pairs);
    auto launch = [&](auto kernel, bool (&done)[64]) {
        if (const int arc = ensure_dynamic_smem(kernel, kSmemBytes, done)) return arc;
        launch_pdl(kernel, dim3(grid), dim3(kThreads), kSmemBytes, st, maps, plan, prm);
        return launch_status();
    };
    static bool done[2][64] = {};
    return forward ? launch(so2_conv_pair_kernel<kForwardKind>, done[1]) : launch(so2_conv_pair_kernel<kPlainKind>, done[0]);
}

}  // namespace fused
}  // namespace fcb200
