// One launch per SO(2) convolution: a persistent CTA takes 128-edge row tiles and walks the output column tiles of the
// convolution's m-blocks (each with its own slice of the input columns, weight matrix and K extent), with the gate
// activation -- or its derivative -- applied in the epilogue, so that the convolution output never makes a round trip
// through memory as float32 just to be gated:
//
//   conv 1 forward : A = rotated+radial-scaled rows (hi, lo planes)  ->  tiles [gate scalars | rows]
//                    gate tiles  : raw float32 into y; their sigmoid stays in the epilogue's registers for the rows of that
//                                  degree, which follow
//                    row tiles   : row 0 -> v * sigmoid(v); row (l, m) -> v * sigmoid(gate[l-1]); written as the
//                                  (hi, lo) half planes conv 2 reads; raw y rows are stored only when the backward
//                                  pass will want them
//   conv 2 forward : plain float32 output (messages)
//   conv 2 backward: A = message gradient planes -> tiles = rows of the gate output's gradient; the epilogue
//                    reads the kept y, writes the gradient of the conv-1 output as (hi, lo) planes and sums the
//                    gate-scalar gradients over the rows of a degree in registers (the tiles of a degree are
//                    consecutive: the first resets the sums, the last writes them into the planes); where the gated rows
//                    were kept as planes it reads those instead of the rows of y, which are then not written at all
//                    (4 of 23 KB an edge that conv 1 moves at lmax 2; 2 000 atoms of alloy 10.35 -> 10.15 ms, 25 000 of water 124.4 -> 121.5).
//                    Planes hold 22 bits of y sigmoid(g), below 6e-5 1.5e-11 absolute, what conv 2 itself has read.  Forces against
//                    float64 of 105 evaluations (lmax 2 and 4; gates half open, closed to 2e-9, spread over both): in none of ten
//                    groups is the mean error more than 1.002 times that of float32 rows; it is the larger one in 53.
//   conv 1 backward: plain float32 output (gradient of the rotated rows)
//
// Replaces SO2_Convolution.forward + GateActivation.forward of the reference
// (src/fairchem/core/models/uma/nn/so2_layers.py:600-647, src/fairchem/core/models/uma/nn/activation.py:146-165)
// and their autograd twins.  Arithmetic and accumulators are those of gemm_f16x2_presplit_kernel.
//
// What bounds it, and the layout that follows.  Per 64-deep k-step a 128 x 128 tile takes 768 cycles of MMA and 64 KiB of
// operands: 128-byte swizzle (the MMAs alone issue 1736 TFLOP/s from it, 1516 from the 64-byte one), 64-deep stages, three of
// them (192 KiB; two: 1250 against 1527 TFLOP/s), which leaves 32 KiB for the epilogue, one 4 KiB tile for each of its eight
// warps.  A warp turns its 32 x 32 accumulator block in that tile from a row per lane to whole lines per instruction and does
// everything else on registers and global memory directly.
// The products are issued by one lane of a warp that walks the loop as one; from a branch of a single lane each took some 110
// cycles to issue whatever its shape, and a k-step 1125.  24 k-steps of one row tile (radial output layer's backward), us:
// 17.8 -> 15.2 with 128 columns an item, 16.2 -> 11.3 with 32.
// At size a launch runs at the power cap and its energy is what there is to save (see so2_conv_pair.cu); few row tiles are
// bound by the chain of k-steps of one item, hence items of 64 or 32 columns there.
#include "so2_conv.cuh"

namespace fcb200 {
namespace fused {

// A work item is one row tile times one group of consecutive tiles [begin[g], begin[g + 1]): what has to pass through one
// CTA in order.  See group_tiles() on the host.
struct Plan {
    Order order;
    int16_t begin[kMaxPlan + 1];
    Tile t[kMaxPlan];
};

// NB: columns of a work item, 128, or 64 or 32 where few row tiles would leave SMs without work.
template <int NB> constexpr int kStages = NB == 128 ? 3 : NB == 64 ? 4 : 5;
template <int NB> constexpr int kStageBytes = 2 * kPart + 2 * NB * KB * 2;  // A_hi | A_lo | W_hi | W_lo
constexpr int kEpiWarps = 8;
constexpr int kThreads = 128 + 32 * kEpiWarps;       // warp 0 TMA, warp 1 MMA, 2-3 idle, warps 4-11 epilogue
// Registers: launched with 168 a thread (12 warps on 4 schedulers); the first warpgroup gives up what the two epilogue
// warpgroups take, 128 * 40 + 256 * 232 = 384 * 168.
constexpr int kIdleRegs = 40, kEpiRegs = 232;
static_assert(128 * kIdleRegs + 32 * kEpiWarps * kEpiRegs <= kThreads * 168, "register split");
template <int NB> constexpr int kAccCols = 2 * NB;  // main columns [0, NB), corrections [NB, 2 NB); double buffered
template <int NB> constexpr int kEpiBytes = (NB == 32 ? kEpiWarps / 2 : kEpiWarps) * 4096;
template <int NB> constexpr int kSmemBytes = kStages<NB> * kStageBytes<NB> + kEpiBytes<NB> + 1024 + 256;

__device__ __forceinline__ void store_split(__half* hi, __half* lo, int off, f32x2 o0, f32x2 o1, bool in, __half2& top) {
    uint2 h, l;
    split2(o0, h.x, l.x, top);
    split2(o1, h.y, l.y, top);
    if (in) {
        __stcs(reinterpret_cast<uint2*>(hi + off), h);  // streamed: not read again by this kernel
        __stcs(reinterpret_cast<uint2*>(lo + off), l);
    }
}
__device__ __forceinline__ void store_pair(float* p, f32x2 a, f32x2 b) {
    asm volatile("st.global.cs.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void load_pair(const float* p, f32x2& a, f32x2& b) {
    asm volatile("ld.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p));
}

// Epilogue warps 4..11: warp w reads TMEM lanes [32 (w % 4), +32) -- one accumulator row per lane -- and takes the columns
// [64 h, 64 h + 64) of every tile, h = (w - 4) / 4, in two chunks of 32.  A chunk is turned in the warp's shared tile to
// "lane = row 4 i + lane / 8, columns 4 (lane % 8)": 128-byte lines per row for every global access, and the same
// (row, column) in the same thread for every tile, so gates and gate-gradient sums stay in registers.
// Narrow items have one chunk a warp (NB 64) or for the four warps of the first half alone (NB 32).
template <int KIND, int NB>
__device__ __forceinline__ void epilogue(const Plan& plan, const Params& prm, uint32_t tmem_base, uint32_t tile,
                                         uint32_t tfull0, uint32_t tempty0, volatile int* abort_flag, volatile int* range_flag) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = warp & 3, half = (warp - 4) >> 2;
    constexpr int kChunks = NB == 128 ? 2 : 1, kSubs = BN / NB;
    const int base = half * kChunks * 32;  // of this warp's columns in an item
    const int rr = lane >> 3, c4 = (lane & 7) * 4;
    const float a_scale = prm.a_scale ? *prm.a_scale : 1.0f;
    const float o_scale = prm.o_scale ? *prm.o_scale : 1.0f;
    __half2 top = __floats2half2_rn(0.f, 0.f);
    // per chunk and row: forward: o_scale * sigmoid of the gate; backward: gate-gradient sums
    constexpr bool kBackward = KIND >= kBackwardKind, kFromPlanes = KIND == kPlanesKind;
    f32x2 keepv[KIND == kPlainKind ? 1 : kChunks][16];
    // Loads run one chunk ahead where the registers allow it: the second chunk's accumulator columns without a backward
    // input, else the y rows of the next chunk.
    constexpr bool kAhead = !kBackward;
    f32x2 yv[kBackward ? 16 : 1] = {};  // from planes: hi and lo of four columns
    f32x2 sg[kBackward ? kChunks : 1][16];  // backward: o_scale * sigmoid of the degree's gate, made at its first row; row 0: the slope
    auto slot = [&](int i) { return tile + (uint32_t)((rr + 4 * i) * 128 + (((lane & 7) ^ ((rr + 4 * i) & 7)) * 16)); };
    auto put = [](uint32_t at, f32x2 a, f32x2 b) { asm volatile("st.shared.v2.b64 [%0], {%1,%2};" ::"r"(at), "l"(a), "l"(b) : "memory"); };
    auto get = [](uint32_t at, f32x2& a, f32x2& b) { asm volatile("ld.shared.v2.b64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "r"(at) : "memory"); };
    // y lines of a backward tile on their way to L2 one tile early (lane = row, a line a chunk)
    auto prefetch = [&](int64_t mt2, int ti2, int first) {
        if constexpr (kBackward) {
            const int64_t row = mt2 * BM + q * 32 + lane;
            if (row < prm.m_total) {
                const Tile& t2 = plan.t[ti2];
                const float* p = prm.y + row * prm.ldy + first;
                if (kFromPlanes && t2.mode == kGatedBwd) {
                    const int64_t at = row * prm.ld_rows + t2.y_col + first;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(prm.rows_hi + at));
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(prm.rows_lo + at));
                } else {
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(p + t2.y_col));
                    if (kChunks == 2) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + t2.y_col + 32));
                }
                if (t2.flags & kFirst) {
                    p += t2.gate_col;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
                    if (kChunks == 2) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 32));
                }
            }
        }
    };
    uint32_t r[kAhead ? 32 : 1], c[kAhead ? 32 : 1];
    int64_t tcount = 0, mt;
    int g;
    for (int64_t n = 0; plan.order.item(n, gridDim.x, blockIdx.x, mt, g); ++n) {
        const int col0 = NB == 128 ? half * 64 : g % kSubs * NB + base;  // of this warp's first chunk in a listed tile
        if (NB < 128) g /= kSubs;
        const int64_t row0 = mt * BM + q * 32;
        const int live = (int)(prm.m_total - row0 < 32 ? prm.m_total - row0 : 32);  // rows of this warp inside the matrix
        // 32 rows of at most 32 767 columns: offsets inside a warp's block fit 32 bits
        float* const yrow = prm.y + (row0 + rr) * prm.ldy + c4;
        __half* const ohi = prm.o_hi + (row0 + rr) * prm.ldo + c4;
        __half* const olo = prm.o_lo + (row0 + rr) * prm.ldo + c4;
        auto fetch = [&](int y_col, int c2) {
            if constexpr (kFromPlanes) {
                const int64_t at = (row0 + rr) * prm.ld_rows + y_col + col0 + c2 * 32 + c4;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    yv[2 * i] = yv[2 * i + 1] = 0;
                    if (rr + 4 * i < live) {
                        yv[2 * i] = *reinterpret_cast<const uint64_t*>(prm.rows_hi + at + 4 * i * prm.ld_rows);
                        yv[2 * i + 1] = *reinterpret_cast<const uint64_t*>(prm.rows_lo + at + 4 * i * prm.ld_rows);
                    }
                }
            } else if constexpr (kBackward) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    yv[2 * i] = yv[2 * i + 1] = 0;
                    if (rr + 4 * i < live) load_pair(yrow + 4 * i * prm.ldy + y_col + col0 + c2 * 32, yv[2 * i], yv[2 * i + 1]);
                }
            }
        };
        auto fetch_of = [&](const Tile& t2, int c2) {
            if (t2.mode == kGatedBwd) fetch(t2.y_col, c2);
        };
        fetch_of(plan.t[plan.begin[g]], 0);
        for (int ti = plan.begin[g]; ti < plan.begin[g + 1]; ++ti, ++tcount) {
            const Tile& t = plan.t[ti];
            const int mode = t.mode;
            const int buf = (int)(tcount & 1);
            const uint32_t use = (uint32_t)((tcount >> 1) & 1);
            if constexpr (kBackward) {
                int64_t mt2;
                int g2;
                if (ti + 1 < plan.begin[g + 1]) prefetch(mt, ti + 1, col0);
                else if (plan.order.item(n + 1, gridDim.x, blockIdx.x, mt2, g2)) prefetch(mt2, plan.begin[g2 / kSubs], NB == 128 ? col0 : g2 % kSubs * NB + base);
            }
            const bool gate_silu = (t.flags & kGateSilu) != 0;
            // What the rows that follow are multiplied by, made while the tensor core works on the tile.  The values pass
            // through the thread's own slots of the shared tile so that the sigmoids are a loop: unrolled for both chunks,
            // and with row 0 and the gate's gradient unrolled too, the code of a tile outgrew the instruction cache and a
            // quarter of the epilogue's stalls were instruction fetches (gated backward launches of an evaluation, 62 118 edges:
            // 1.40 -> 1.26 ms; 775 000: 18.9 -> 17.3).
            if constexpr (kBackward) {
                if (mode == kSiluBwd || (t.flags & kFirst)) {
                    const bool slope = mode == kSiluBwd;
                    const float* from = yrow + (slope ? t.y_col : t.gate_col) + col0;
#pragma unroll
                    for (int i = 0; i < 8 * kChunks; ++i) {
                        f32x2 &a = sg[i >> 3][2 * (i & 7)], &b = sg[i >> 3][2 * (i & 7) + 1];
                        a = b = 0;
                        if (rr + 4 * (i & 7) < live) load_pair(from + 4 * (i & 7) * prm.ldy + (i >> 3) * 32, a, b);
                    }
                    auto factor = [&](float v) {
                        float s = sigmoid_f(v);
                        if (slope) s = s * (1.f + v * (1.f - s));
                        else if (gate_silu) s = sigmoid_f(v * s);
                        return o_scale * s;
                    };
#pragma unroll
                    for (int c2 = 0; c2 < kChunks; ++c2) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) put(slot(i), sg[c2][2 * i], sg[c2][2 * i + 1]);
#pragma unroll 1
                        for (int i = 0; i < 8; ++i) {
                            f32x2 a, b;
                            get(slot(i), a, b);
                            put(slot(i), map2(a, factor), map2(b, factor));
                        }
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            get(slot(i), sg[c2][2 * i], sg[c2][2 * i + 1]);
                            keepv[c2][2 * i] = keepv[c2][2 * i + 1] = 0;
                        }
                    }
                    __syncwarp();  // before other lanes' accumulator rows go to these slots
                }
            }
            bool ok = mbar_wait(tfull0 + 8u * buf, use, abort_flag);
            ok = __all_sync(kFull, ok);
            if (!ok) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float out_scale = 1.0f / (a_scale * prm.w_scale[t.w]);  // a power of two: scaling after the sum is exact
            const f32x2 os2 = pack(out_scale, out_scale);
            const float* bias = prm.bias[t.w];
            const uint32_t acc = tmem_base + (uint32_t)(buf * kAccCols<NB> + base) + ((uint32_t)(q * 32) << 16);
            if constexpr (kAhead) {
                FCB_TMEM_LD32(r, acc);
                FCB_TMEM_LD32(c, acc + (uint32_t)NB);
            }
#pragma unroll
            for (int c2 = 0; c2 < kChunks; ++c2) {
                const int col = col0 + c2 * 32;  // within the tile
                // 1. accumulator -> shared tile, row `lane`
                f32x2 poison = 0;  // becomes NaN if any value is inf or NaN (an overflowed half upstream)
                auto stage4 = [&](int v4, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3, uint32_t c0, uint32_t c1, uint32_t c2_, uint32_t c3) {
                    const f32x2 lo = pack(1.0f / kLoScale, 1.0f / kLoScale);
                    const f32x2 v01 = fma2(pack(__uint_as_float(c0), __uint_as_float(c1)), lo, pack(__uint_as_float(r0), __uint_as_float(r1)));
                    const f32x2 v23 = fma2(pack(__uint_as_float(c2_), __uint_as_float(c3)), lo, pack(__uint_as_float(r2), __uint_as_float(r3)));
                    if (KIND == kPlainKind || mode == kPlain) poison = fma2(v01, 0, fma2(v23, 0, poison));
                    const uint32_t dst = tile + (uint32_t)(lane * 128 + ((v4 ^ (lane & 7)) * 16));
                    asm volatile("st.shared.v2.b64 [%0], {%1,%2};" ::"r"(dst), "l"(v01), "l"(v23) : "memory");
                };
                if constexpr (kAhead) {
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int v = 0; v < 8; ++v)
                        stage4(v, r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3], c[4 * v], c[4 * v + 1], c[4 * v + 2], c[4 * v + 3]);
                    if (c2 + 1 < kChunks) {
                        FCB_TMEM_LD32(r, acc + 32u);
                        FCB_TMEM_LD32(c, acc + (uint32_t)(NB + 32));
                    }
                } else {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t rh[16], ch[16];
                        FCB_TMEM_LD16(rh, acc + (uint32_t)(c2 * 32 + 16 * h));
                        FCB_TMEM_LD16(ch, acc + (uint32_t)(NB + c2 * 32 + 16 * h));
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int v = 0; v < 4; ++v)
                            stage4(4 * h + v, rh[4 * v], rh[4 * v + 1], rh[4 * v + 2], rh[4 * v + 3], ch[4 * v], ch[4 * v + 1], ch[4 * v + 2], ch[4 * v + 3]);
                    }
                }
                if (c2 == kChunks - 1) {  // hand the accumulator back to the MMA thread
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    mbar_arrive(tempty0 + 8u * buf);
                }
                {
                    float p0, p1;
                    unpack(poison, p0, p1);
                    if (!(p0 + p1 == 0.f) && lane < live) *range_flag = 1;
                }
                __syncwarp();
                // 2. whole lines: the mode's arithmetic and its stores
                float4 b = f4zero();
                if (bias) b = ld4(bias + t.w_row + col + c4);
                const f32x2 b01 = pack(b.x, b.y), b23 = pack(b.z, b.w);
                // body(i, x01, x23, in): row rr + 4 i of the chunk, four columns
                auto row_of = [&](int i, f32x2 x0, f32x2 x1, auto&& body) {
                    if constexpr (kBackward) body(i, mul2(x0, os2), mul2(x1, os2), rr + 4 * i < live);
                    else body(i, fma2(x0, os2, b01), fma2(x1, os2, b23), rr + 4 * i < live);
                };
                // Shared reads of four rows first: a read keeps its place behind another row's stores, and so behind its
                // arithmetic (gated backward launches of an evaluation, 155 000 edges: 3.45 -> 3.17 ms).
                auto rows = [&](auto&& body) {
#pragma unroll
                    for (int i0 = 0; i0 < 8; i0 += 4) {
                        f32x2 x[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) get(slot(i0 + i), x[2 * i], x[2 * i + 1]);
#pragma unroll
                        for (int i = 0; i < 4; ++i) row_of(i0 + i, x[2 * i], x[2 * i + 1], body);
                    }
                };
                auto loop = [&](auto&& body) {
#pragma unroll 2
                    for (int i = 0; i < 8; ++i) {
                        f32x2 x0, x1;
                        get(slot(i), x0, x1);
                        row_of(i, x0, x1, body);
                    }
                };
                float* const yo = yrow + col;
                __half *const ph = ohi + t.out_col + col, *const pl = olo + t.out_col + col;
                auto gate_of = [&](float v) { return o_scale * sigmoid_f(gate_silu ? v * sigmoid_f(v) : v); };
                if (KIND == kPlainKind || mode == kPlain) {
                    const bool inside = t.out_col + col + c4 < prm.y_cols;
                    auto store = [&](int i, f32x2 x0, f32x2 x1, bool in) {
                        if (in && inside) store_pair(yo + 4 * i * prm.ldy + t.out_col, x0, x1);
                    };
                    if constexpr (KIND == kForwardKind) {  // sigmoids in a loop for the code's size (155 000 edges 4.67 -> 4.55 ms, 3 240: 0.45 -> 0.43)
                        loop([&](int i, f32x2 x0, f32x2 x1, bool in) {
                            store(i, x0, x1, in);
                            put(slot(i), map2(x0, gate_of), map2(x1, gate_of));
                        });
                        if (t.flags & kGateSrc) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) get(slot(i), keepv[c2][2 * i], keepv[c2][2 * i + 1]);
                        }
                    } else {
                        rows(store);
                    }
                } else if constexpr (KIND == kForwardKind) {
                    const bool keep = (t.flags & kKeep) != 0;
                    if (mode == kSilu) {
                        auto sig = [&](float v) { return o_scale * sigmoid_f(v); };
                        loop([&](int i, f32x2 x0, f32x2 x1, bool in) {
                            if (in && keep) store_pair(yo + 4 * i * prm.ldy + t.y_col, x0, x1);
                            store_split(ph, pl, 4 * i * prm.ldo, mul2(x0, map2(x0, sig)), mul2(x1, map2(x1, sig)), in, top);
                        });
                    } else {
                        rows([&](int i, f32x2 x0, f32x2 x1, bool in) {
                            if (in && keep) store_pair(yo + 4 * i * prm.ldy + t.y_col, x0, x1);
                            store_split(ph, pl, 4 * i * prm.ldo, mul2(x0, keepv[c2][2 * i]), mul2(x1, keepv[c2][2 * i + 1]), in, top);
                        });
                    }
                } else {
                    rows([&](int i, f32x2 x0, f32x2 x1, bool in) {
                        f32x2 y0 = yv[2 * i], y1 = yv[2 * i + 1];
                        if constexpr (kFromPlanes) join2(yv[2 * i], yv[2 * i + 1], y0, y1);
                        keepv[c2][2 * i] = fma2(x0, y0, keepv[c2][2 * i]);  // row 0: not used
                        keepv[c2][2 * i + 1] = fma2(x1, y1, keepv[c2][2 * i + 1]);
                        store_split(ph, pl, 4 * i * prm.ldo, mul2(x0, sg[c2][2 * i]), mul2(x1, sg[c2][2 * i + 1]), in, top);
                    });
                    if (t.flags & kLast) {
                        const float inv = 1.0f / o_scale;
                        auto dsig = [&](float v) { return kFromPlanes ? o_scale - v : v * (1.f - v * inv); };  // o_scale * sigmoid', or that over sigmoid
                        auto dsilu = [&](float v) {
                            const float q = sigmoid_f(v);
                            return q * (1.f + v * (1.f - q));
                        };
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            put(slot(i), mul2(keepv[c2][2 * i], map2(sg[c2][2 * i], dsig)), mul2(keepv[c2][2 * i + 1], map2(sg[c2][2 * i + 1], dsig)));
#pragma unroll 1
                        for (int i = 0; i < 8; ++i) {
                            f32x2 d0, d1;
                            get(slot(i), d0, d1);
                            const bool in = rr + 4 * i < live;
                            if (gate_silu) {
                                f32x2 g0 = 0, g1 = 0;
                                if (in) load_pair(yo + 4 * i * prm.ldy + t.gate_col, g0, g1);
                                d0 = mul2(d0, map2(g0, dsilu)), d1 = mul2(d1, map2(g1, dsilu));
                            }
                            store_split(ohi + t.gate_col + col, olo + t.gate_col + col, 4 * i * prm.ldo, d0, d1, in, top);
                        }
                    }
                }
                if (c2 + 1 < kChunks) fetch_of(t, 1);
                else if (ti + 1 < plan.begin[g + 1]) fetch_of(plan.t[ti + 1], 0);
                __syncwarp();  // the shared tile is free again
            }
        }
    }
    if (!(__half2float(__hmax_nan(__low2half(top), __high2half(top))) <= kHalfMax)) *range_flag = 1;  // inf or NaN
}

template <int KIND, int NB>
__global__ void __launch_bounds__(kThreads, 1)
    so2_conv_fused_kernel(const __grid_constant__ CUtensorMap map_ahi, const __grid_constant__ CUtensorMap map_alo,
                          const __grid_constant__ CUtensorMap map_whi0, const __grid_constant__ CUtensorMap map_wlo0,
                          const __grid_constant__ CUtensorMap map_whi1, const __grid_constant__ CUtensorMap map_wlo1,
                          const __grid_constant__ CUtensorMap map_whi2, const __grid_constant__ CUtensorMap map_wlo2,
                          const __grid_constant__ Plan plan, const __grid_constant__ Params prm) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    constexpr int kRing = kStages<NB>, kTmemCols = 2 * kAccCols<NB>;
    const uint32_t epi_base = base + kRing * kStageBytes<NB>;
    const uint32_t bar_base = epi_base + kEpiBytes<NB>;
    // barrier block: full[ring] | empty[ring] | tmem_full[2] | tmem_empty[2] | tmem slot, abort flag, range flag
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kRing + s); };
    auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * kRing + b); };
    auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * kRing + 2 + b); };
    uint8_t* const bar_generic = smem_raw + (bar_base - smem_u32(smem_raw));
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_generic + 8 * (2 * kRing + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_generic + 8 * (2 * kRing + 4) + 4);
    volatile int* range_flag = reinterpret_cast<volatile int*>(bar_generic + 8 * (2 * kRing + 4) + 8);
    // A_hi, A_lo, W_hi, W_lo of a stage
    auto part_addr = [&](int s, int which) { return base + s * kStageBytes<NB> + (which < 2 ? which * kPart : 2 * kPart + (which - 2) * (NB * KB * 2)); };

    const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kRing; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull_bar(b), 1);
            mbar_init(tempty_bar(b), NB == 32 ? 128 : 32 * kEpiWarps);
        }
        *abort_flag = 0;
        *range_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)),
                     "r"((uint32_t)kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 64) {
        prefetch_map(&map_ahi), prefetch_map(&map_alo);
        prefetch_map(&map_whi0), prefetch_map(&map_wlo0), prefetch_map(&map_whi1), prefetch_map(&map_wlo1), prefetch_map(&map_whi2), prefetch_map(&map_wlo2);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    pdl_sync();  // barriers and tensor memory are set up while the predecessor finishes

    if (warp >= 4) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpiRegs));
        if (NB > 32 || warp < 8)
            epilogue<KIND, NB>(plan, prm, tmem_base, epi_base + (uint32_t)((warp - 4) * 4096), tfull_bar(0), tempty_bar(0), abort_flag, range_flag);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIdleRegs));
        if (warp == 0 && lane == 0) {
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            // an A tile is fetched again for each of the output tiles of its m-block, the weights by every CTA: keep
            // both in L2 ahead of the streamed outputs
            const uint64_t keep = l2_policy_evict_last();
            int64_t mt;
            int g;
            for (int64_t n = 0; ok && plan.order.item(n, gridDim.x, blockIdx.x, mt, g); ++n) {
                const int row = (int)(mt * BM), sub = NB == 128 ? 0 : g % (BN / NB) * NB;
                if (NB < 128) g /= BN / NB;
                for (int ti = plan.begin[g]; ti < plan.begin[g + 1] && ok; ++ti) {
                    const Tile& t = plan.t[ti];
                    const CUtensorMap* whi = t.w == 0 ? &map_whi0 : (t.w == 1 ? &map_whi1 : &map_whi2);
                    const CUtensorMap* wlo = t.w == 0 ? &map_wlo0 : (t.w == 1 ? &map_wlo1 : &map_wlo2);
                    const int num_kb = (t.k + KB - 1) / KB;
                    for (int kb = 0; kb < num_kb; ++kb) {
                        ok = mbar_wait(empty_bar(s), ph, abort_flag);
                        if (!ok) break;
                        mbar_expect_tx(full_bar(s), kStageBytes<NB>);
                        tma_load_2d_hint(part_addr(s, 0), &map_ahi, t.a_col + kb * KB, row, full_bar(s), keep);
                        tma_load_2d_hint(part_addr(s, 1), &map_alo, t.a_col + kb * KB, row, full_bar(s), keep);
                        tma_load_2d_hint(part_addr(s, 2), whi, kb * KB, t.w_row + sub, full_bar(s), keep);
                        tma_load_2d_hint(part_addr(s, 3), wlo, kb * KB, t.w_row + sub, full_bar(s), keep);
                        if (++s == kRing) s = 0, ph ^= 1;
                    }
                }
            }
        }
        // All lanes of the warp walk the loop and one issues: addresses and descriptors are then the same in every lane, which
        // is where the instruction takes them from.  (Issued from a branch of lane 0 alone, a product cost some 110 cycles
        // whatever its shape, and a 64-deep step 1125 instead of the 768 its products take.)
        if (warp == 1) {
            int s = 0, buf = 0, g;
            uint32_t ph = 0, free_ph = 1;
            int64_t mt;
            bool ok = true;
            const uint64_t desc0 = smem_desc128(base);
            for (int64_t n = 0; ok && plan.order.item(n, gridDim.x, blockIdx.x, mt, g); ++n) {
                if (NB < 128) g /= BN / NB;
                for (int ti = plan.begin[g]; ti < plan.begin[g + 1] && ok; ++ti) {
                    const int k = plan.t[ti].k, num_kb = (k + KB - 1) / KB;
                    ok = mbar_wait_warp(tempty_bar(buf), free_ph, abort_flag);  // epilogue has drained this accumulator
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t acc = tmem_base + (uint32_t)(buf * kAccCols<NB>);
                    for (int kb = 0; kb < num_kb; ++kb) {
                        ok = mbar_wait_warp(full_bar(s), ph, abort_flag);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        // W_hi | W_lo are adjacent: one MMA of 2 NB columns on a_hi gives a_hi*w_hi (main accumulator) and
                        // a_hi*w_lo (correction accumulator); one of NB columns adds a_lo*w_hi to the correction
                        const uint64_t da = desc0 + (uint64_t)(s * (kStageBytes<NB> >> 4));
                        const int steps = (k - kb * KB + 15) / 16;  // columns past k belong to a neighbour: not multiplied
                        if (elect_one()) {
                            constexpr uint64_t kLo = kPart >> 4, kW = 2 * kLo;
                            umma_one<2 * NB, false>(acc, da, da + kW, kb > 0);
                            umma_one<NB, true>(acc + NB, da + kLo, da + kW, 1u);
                            if (steps >= KB / 16) {
#pragma unroll
                                for (uint64_t j = 2; j < KB / 8; j += 2) {
                                    umma_one<2 * NB, true>(acc, da + j, da + j + kW, 1u);
                                    umma_one<NB, true>(acc + NB, da + j + kLo, da + j + kW, 1u);
                                }
                            } else {
                                for (int j = 1; j < steps; ++j) {
                                    const uint64_t d = da + (uint64_t)(2 * j);
                                    umma_one<2 * NB, true>(acc, d, d + kW, 1u);
                                    umma_one<NB, true>(acc + NB, d + kLo, d + kW, 1u);
                                }
                            }
                            umma_commit(empty_bar(s));
                        }
                        __syncwarp();
                        if (++s == kRing) s = 0, ph ^= 1;
                    }
                    if (ok && elect_one()) umma_commit(tfull_bar(buf));
                    __syncwarp();
                    if (buf) free_ph ^= 1;
                    buf ^= 1;
                }
            }
        }
    }

    settle(abort_flag);
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
    }
    if (threadIdx.x == 0 && prm.status) {
        if (*abort_flag) atomicExch(prm.status, 1);
        else if (*range_flag) atomicCAS(prm.status, 0, 2);
    }
}

// 2-D row-major half matrix [rows, cols], row stride ld elements; box = 64 columns, 128-byte swizzle
static int map_half(CUtensorMap* map, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return FCB200_EINVAL;
    cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t gstride[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)KB, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? FCB200_OK : FCB200_EINVAL;
}

// ---- work items ----------------------------------------------------------------------------------------------------
// How a tile list is cut into groups (Plan::groups); a CTA takes (row tile, group) items in turn.
//   natural  what shares nothing is apart: every plain tile, row 0, and the rows of a degree with their gate tile (forward)
//            or their gate-gradient sum (backward)
//   fine     forward gated rows one by one, each after its own copy of the gate tile (the gate is computed again)
//   pair     natural groups on CTA pairs, tiles that read the same columns side by side (so2_conv_pair.cu)
enum Grouping { kAuto = 0, kNatural = 1, kFine = 2, kPair = 3 };

struct Groups {
    int n = 0;           // tiles
    int groups = 0;
    int16_t begin[kMaxPlan + 1] = {};
    int16_t tile[kMaxPlan] = {};  // index into the caller's list
    bool ok = true;
};

// Units of K: what a tile's K extent counts in items of 128, 64 and 32 columns (percent), a tile's fixed share (epilogue, ring
// start-up), the same with the gate's backward, and of a tile on a pair of CTAs; from launches of one row tile.
constexpr int kStepCost[3] = {100, 70, 58}, kTileCost[3] = {192, 150, 130}, kBackwardTileCost[3] = {416, 183, 143}, kPairTileCost = 250;

static Groups group_tiles(const Tile* t, int n, int rot_begin, int how) {
    Groups g;
    auto put = [&](int i) {
        if (g.n >= kMaxPlan) {
            g.ok = false;
            return;
        }
        g.tile[g.n++] = (int16_t)i;
    };
    auto close = [&] { g.begin[++g.groups] = (int16_t)g.n; };
    auto gate_of = [&](int col) {
        for (int i = 0; i < rot_begin; ++i)
            if (t[i].mode == kPlain && t[i].out_col == col) return i;
        return -1;
    };
    bool done[kMaxTiles] = {};
    for (int i = 0; i < n && g.ok; ++i) {
        if (done[i] || (t[i].flags & kGateSrc)) continue;
        if (t[i].mode == kGated) {
            const int gate = gate_of(t[i].gate_col);
            if (gate < 0) {
                g.ok = false;
                break;
            }
            bool opened = false;
            for (int j = i; j < n; ++j) {
                if (t[j].mode != kGated || t[j].gate_col != t[i].gate_col) continue;
                if (!opened || how == kFine) {
                    if (opened) close();
                    put(gate);
                    opened = true;
                }
                put(j);
                done[j] = true;
            }
        } else if (t[i].mode == kGatedBwd) {
            for (int j = i; j < n; ++j) {
                put(j);
                done[j] = true;
                if (t[j].flags & kLast) break;
            }
        } else {
            put(i);
        }
        close();
    }
    return g;
}

// The natural groups with row 0 in the group of degree 1: two groups of about the same length at lmax 2, which then read the
// same input columns at the same time.
static Groups with_row0(const Tile* t, const Groups& g) {
    Groups j;
    j.ok = g.ok && g.groups > 1 && g.begin[1] == 1 && (t[g.tile[0]].mode == kSilu || t[g.tile[0]].mode == kSiluBwd) && g.begin[2] > 2;
    if (!j.ok) return j;
    // forward behind the tiles that read the same columns; backward in front, since its factors take the place of the gate's
    int at = 1;
    if (t[g.tile[0]].mode == kSilu)
        while (at < g.begin[2] && t[g.tile[at]].a_col == t[g.tile[0]].a_col) ++at;
    for (int i = 1; i < at; ++i) j.tile[j.n++] = g.tile[i];
    j.tile[j.n++] = g.tile[0];
    for (int i = at; i < g.n; ++i) j.tile[j.n++] = g.tile[i];
    for (int i = 1; i < g.groups; ++i) j.begin[++j.groups] = g.begin[i + 1];
    return j;
}

// Natural groups for CTA pairs: tiles of a group two by two where they follow one another and read the same columns; groups
// of a single tile that no order binds to others are joined the same way.
struct PairGroups {
    PairPlan plan{};
    int cost[kMaxTiles] = {};
};
static PairGroups pair_tiles(const Tile* t, const Groups& g) {
    PairGroups out;
    PairPlan& p = out.plan;
    int n = 0, groups = 0;
    auto joins = [&](const PairTile& a, const Tile& b) { return a.n == 1 && a.a_col == b.a_col && a.k == b.k && a.w == b.w; };
    bool open = false;  // the last group is one lone tile
    for (int i = 0; i < g.groups; ++i) {
        const bool lone = g.begin[i + 1] - g.begin[i] == 1;
        if (!(lone && open && joins(p.t[n - 1], t[g.tile[g.begin[i]]]))) p.begin[groups++] = (int16_t)n;
        for (int j = g.begin[i]; j < g.begin[i + 1]; ++j) {
            const Tile& s = t[g.tile[j]];
            if (n == p.begin[groups - 1] || !joins(p.t[n - 1], s)) {
                p.t[n] = PairTile{};
                p.t[n].a_col = s.a_col, p.t[n].k = s.k, p.t[n].w = s.w;
                ++n;
            }
            PairTile& d = p.t[n - 1];
            d.w_row[d.n] = s.w_row, d.out_col[d.n] = s.out_col, d.mode[d.n] = s.mode, d.y_col[d.n] = s.y_col, d.flags[d.n] = s.flags;
            ++d.n;
        }
        open = lone && n - p.begin[groups - 1] == 1 && p.t[n - 1].n == 1;
        p.begin[groups] = (int16_t)n;
    }
    p.order.groups = groups;
    for (int i = 0; i < groups; ++i)
        for (int j = p.begin[i]; j < p.begin[i + 1]; ++j) out.cost[i] += p.t[j].n == 2 ? 2 * (8 * p.t[j].k / 10 + kPairTileCost) : p.t[j].k + kPairTileCost;
    return out;
}

// Longest of `units` CTAs or pairs, in units of K; an item's group is one of `subs` parts of a group of tiles.
static int64_t makespan(const Order& order, const int* cost, int subs, int units) {
    const int64_t items = order.rows * order.groups;
    int64_t total = 0, most = 0;
    for (int i = 0; i < order.groups; ++i) total += cost[i / subs], most = cost[i / subs] > most ? cost[i / subs] : most;
    if (units > 256 || items > 32LL * units) return order.rows * total / units + most;
    if (items <= units) return most;
    int64_t sum[256] = {}, worst = 0;
    int unit = 0, step = 1, row = 0, group = 0;
    for (int64_t i = 0; i < items; ++i) {
        sum[unit] += cost[group / subs];
        worst = sum[unit] > worst ? sum[unit] : worst;
        unit += step;
        if (unit == units || unit < 0) {  // the next round goes back
            unit -= step;
            step = -step;
        }
        if (order.by_group ? ++row == order.rows : ++group == order.groups) {
            group = order.by_group ? group + 1 : 0;
            row = 0;
        }
    }
    return worst;
}

// The order of a launch's items and its makespan.  perm: the groups by falling cost.  Group by group an A tile leaves L2
// between its groups when there are many rows, so that has to gain more than the extra reads cost (us row by row / group by group,
// lmax 2: first convolution, 7 200 rows 75.7 / 54.9, 14 000 rows 110 / 101, 40 000 rows 271 / 301; second convolution's backward, 7 200 rows 62.7 /
// 35.8, 14 000 rows 99 / 67; second convolution, 5 000 rows 19.0 / 16.9, 14 000 rows 47.1 / 48.6).
static int64_t choose_order(Order& order, int* cost, int* perm, int subs, int units) {
    const int groups = order.groups / subs;
    for (int i = 0; i < groups; ++i) perm[i] = i;
    const int64_t by_row = makespan(order, cost, subs, units), items = order.rows * order.groups;
    if (items > 8LL * units || items <= units) return by_row;
    int sorted[kMaxPlan], at[kMaxPlan];
    for (int i = 0; i < groups; ++i) {
        int j = i;
        for (; j > 0 && cost[i] > sorted[j - 1]; --j) sorted[j] = sorted[j - 1], at[j] = at[j - 1];
        sorted[j] = cost[i], at[j] = i;
    }
    Order other = order;
    other.by_group = 1;
    const int64_t by_group = makespan(other, sorted, subs, units);
    if (100 * by_group >= 96 * by_row) return by_row;
    order = other;
    for (int i = 0; i < groups; ++i) cost[i] = sorted[i], perm[i] = at[i];
    return by_group;
}
static PairPlan reordered(const PairPlan& p, const int* perm) {
    PairPlan q = p;
    int n = 0;
    for (int g = 0; g < p.order.groups; ++g) {
        for (int i = p.begin[perm[g]]; i < p.begin[perm[g] + 1]; ++i) q.t[n++] = p.t[i];
        q.begin[g + 1] = (int16_t)n;
    }
    return q;
}
// Groups on single CTAs, `width` of each tile's 128 columns an item, with the order of their items.
struct Schedule {
    Groups g;
    int width, perm[kMaxPlan];
    Order order;
    int64_t span;
    Schedule(const Groups& groups, const Tile* list, int64_t rows, int w) : g(groups), width(w), order{rows, groups.groups * (BN / w), 0} {
        const int at = w == 128 ? 0 : w == 64 ? 1 : 2;
        int cost[kMaxPlan] = {};
        for (int i = 0; i < g.groups; ++i)
            for (int j = g.begin[i]; j < g.begin[i + 1]; ++j) cost[i] += list[g.tile[j]].k * kStepCost[at] / 100 + (list[g.tile[j]].mode == kGatedBwd ? kBackwardTileCost : kTileCost)[at];
        span = choose_order(order, cost, perm, BN / w, sm_count());
    }
    void fill(Plan& plan, const Tile* list) const {
        plan.order = order;
        int n = 0;
        for (int i = 0; i < g.groups; ++i) {
            for (int j = g.begin[perm[i]]; j < g.begin[perm[i] + 1]; ++j) plan.t[n++] = list[g.tile[j]];
            plan.begin[i + 1] = (int16_t)n;
        }
    }
};

}  // namespace fused
}  // namespace fcb200

using namespace fcb200;

namespace fcb200 {

int so2_conv_fused(const void* a_hi, const void* a_lo, int64_t lda, int64_t a_cols, const void* const* w_hi,
                                     const void* const* w_lo, const int64_t* w_rows, const int64_t* w_cols,
                                     const float* w_scale, const float* const* bias, const int32_t* tiles, int32_t num_tiles,
                                     int32_t rot_begin, float* y, int64_t ldy, int64_t y_cols, void* o_hi, void* o_lo, int64_t ldo, int64_t o_cols,
                                     const float* a_scale, const float* o_scale, int64_t m, int32_t variant, int32_t* status,
                                     void* stream, const __half* rows_hi, const __half* rows_lo, int64_t ld_rows) {
    using namespace fused;
    if (!a_hi || !a_lo || !w_hi || !w_lo || !w_rows || !w_cols || !w_scale || !tiles || !y || m < 0) return FCB200_EINVAL;
    Plan plan{};
    Params prm{};
    Tile list[kMaxTiles] = {};
    const int grouping = variant >> 4;
    if ((variant & 15) > 2 || grouping < kAuto || grouping > kPair) return FCB200_EINVAL;
    if (num_tiles <= 0 || num_tiles > kMaxTiles) return FCB200_ERANGE;
    if (lda % 8 || lda < a_cols || ldy % 4 || ldy < y_cols || y_cols % 4) return FCB200_EINVAL;
    if (!aligned16(a_hi) || !aligned16(a_lo) || !aligned16(y)) return FCB200_EALIGN;
    if (o_hi || o_lo) {
        if (!o_hi || !o_lo || ldo % 8 || ldo < o_cols) return FCB200_EINVAL;
        if (!aligned16(o_hi) || !aligned16(o_lo)) return FCB200_EALIGN;
    }
    if (rot_begin < 0 || rot_begin > num_tiles) return FCB200_EINVAL;
    bool used[3] = {false, false, false};
    bool gated = false, forward = false, backward = false;
    for (int i = 0; i < num_tiles; ++i) {
        Tile& t = list[i];
        const int32_t* d = tiles + 9 * i;
        for (int j = 0; j < 9; ++j)
            if (d[j] < 0 || d[j] > 32767) return FCB200_ERANGE;
        t.a_col = d[0], t.k = d[1], t.w = d[2], t.w_row = d[3], t.out_col = d[4], t.mode = d[5], t.y_col = d[6], t.gate_col = d[7];
        t.flags = d[8] & 15;
        if (t.w < 0 || t.w > 2 || !w_hi[t.w] || !w_lo[t.w]) return FCB200_EINVAL;
        if (t.k <= 0 || t.k % 32 || t.k > w_cols[t.w] || t.a_col < 0 || t.a_col % 8 || t.a_col + t.k > a_cols) return FCB200_EINVAL;
        if (t.w_row % BN || t.w_row >= w_rows[t.w]) return FCB200_EINVAL;
        if (t.mode > kGatedBwd || t.mode == 1 || t.out_col % 8) return FCB200_EINVAL;
        const bool split = t.mode >= kSilu;
        if (w_rows[t.w] - t.w_row < BN && (split || w_rows[t.w] % 4 || t.out_col + (w_rows[t.w] - t.w_row) != y_cols)) return FCB200_EINVAL;
        if (split && (!o_hi || t.out_col + BN > o_cols)) return FCB200_EINVAL;
        if (!split && t.out_col + (w_rows[t.w] - t.w_row < BN ? w_rows[t.w] - t.w_row : BN) > y_cols) return FCB200_EINVAL;
        const bool reads_gate = t.mode == kGated || t.mode == kGatedBwd;
        if (reads_gate && (t.gate_col % 4 || t.gate_col + BN > y_cols)) return FCB200_EINVAL;
        const bool uses_y = t.mode == kSiluBwd || t.mode == kGatedBwd || ((t.mode == kSilu || t.mode == kGated) && (t.flags & kKeep));
        if (uses_y && (t.y_col % 4 || t.y_col + BN > (rows_hi && t.mode == kGatedBwd ? ld_rows : y_cols))) return FCB200_EINVAL;
        if (t.mode == kGatedBwd && t.gate_col + BN > o_cols) return FCB200_EINVAL;
        used[t.w] = true;
        gated = gated || t.mode == kGated;
        forward = forward || t.mode == kSilu || t.mode == kGated;
        backward = backward || t.mode == kSiluBwd || t.mode == kGatedBwd;
    }
    if (forward && backward) return FCB200_EINVAL;
    if (rows_hi && (!rows_lo || ld_rows % 4 || ld_rows > 32767 || !aligned16(rows_hi) || !aligned16(rows_lo))) return FCB200_EINVAL;
    if (m == 0) return FCB200_OK;
    for (int i = 0; i < rot_begin && gated; ++i)
        if (list[i].mode == kPlain) {
            list[i].flags |= kGateSrc;
            for (int j = rot_begin; j < num_tiles; ++j)  // what the gate is follows from the rows that use it
                if (list[j].mode == kGated && list[j].gate_col == list[i].out_col) list[i].flags |= list[j].flags & kGateSilu;
        }
    // Row tiles times natural groups are the items: CTAs that run together share an A tile in L2 and the last wave is one
    // group deep, not one list (whole lists, row tile by row tile, took 11 % longer in the second convolution at 131 072 rows, 18 % in
    // the first at 60 000).  Few row tiles leave SMs without work; then the gated rows of a forward list go one by one, and an item
    // takes a part of its tiles' columns, where that shortens the longest CTA by more than the estimate's error.
    // us, replayed from a graph, 128 / 64 / 32 columns: 420 rows of lmax 2, first convolution row by row 19.8 / 15.7 / 14.6, second
    // 8.8 / 7.3 / 6.8, its gated backward from float32 rows 29.0 / 20.1 / 17.5, radial output layer's backward 15.7 / 12.5 / 11.5; 3 000
    // rows 32.4 / 35.8 / 56.3, 13.1 / 13.5 / 20.1, 29.8 / 20.8 / 23.7, 15.9 / 12.8 / 11.8; 7 680 rows, gated backward 36.7 / 42.1 / 54.9.
    const int64_t rows_m = (m + BM - 1) / BM;
    const Groups natural = group_tiles(list, num_tiles, rot_begin, kNatural);
    if (!natural.ok) return FCB200_EINVAL;
    // Where the input does not stay in L2, groups of one row tile that run apart read it from memory again: at 131 072 rows
    // of lmax 2 the first convolution read 1.43 times its input, the second's backward with its y rows 1.25 times; 1.18 and
    // 1.13 times with row 0 in the group of degree 1 (1019 -> 970 us on pairs, 670 -> 627; 25 000 atoms of water 117.2 -> 116.7 ms).
    const Groups joined = with_row0(list, natural);
    const bool spill = m * a_cols * 4 > (64LL << 20) && joined.ok;
    Schedule run(natural, list, rows_m, BN);
    if (spill && grouping != kFine) {
        const Schedule other(joined, list, rows_m, BN);
        if (100 * other.span <= 103 * run.span) run = other;
    }
    if (!backward && grouping == kFine) {
        run = Schedule(group_tiles(list, num_tiles, rot_begin, kFine), list, rows_m, BN);
        if (!run.g.ok) return FCB200_EINVAL;
    }
    if (grouping == kAuto) {
        auto consider = [&](const Groups& g, int width) {
            if (!g.ok || (width < BN && rows_m * g.groups * (BN / width) > 2 * sm_count())) return;
            const Schedule other(g, list, rows_m, width);
            if (10 * other.span < 9 * run.span) run = other;
        };
        const Groups fine = gated ? group_tiles(list, num_tiles, rot_begin, kFine) : Groups{};
        for (int width = BN; width >= 32; width /= 2) {
            if (width < BN) consider(natural, width);
            if (gated) consider(fine, width);
        }
    }
    // On pairs a listed tile costs 0.8 of its K extent where it has a partner, and 250 for the time the tensor core waits for
    // the accumulators; alone a tile costs its K extent and 192.  So long K goes to pairs, the radial output layer (K = 128)
    // and small launches do not.  us, alone / on pairs (seconds of back-to-back launches, at the power cap): first convolution,
    // lmax 2, 20 580 rows 196 / 176, 131 072 rows 1040 / 980; lmax 4, 7 000 rows 229 / 209, 60 000 rows 1796 / 1594; second
    // convolution, lmax 2, 20 580 rows 71 / 74, 131 072 rows 435 / 410; first convolution's backward, 13 000 rows 98 / 96, 131 072
    // rows 940 / 872; radial output layer, 131 072 rows 246 / 259.
    PairGroups two;
    if (!backward && (grouping == kPair || (grouping == kAuto && rows_m >= 8))) {  // the fewest rows: no time for the estimate
        int64_t best = grouping == kPair ? INT64_MAX / 100 : run.span;
        auto consider = [&](const Groups& g, int64_t percent) {
            PairGroups other = pair_tiles(list, g);
            other.plan.order.rows = (m + 2 * BM - 1) / (2 * BM);
            int perm[kMaxPlan];
            const int64_t span = choose_order(other.plan.order, other.cost, perm, 1, sm_count() / 2);
            if (100 * span >= percent * best) return;
            best = span;
            two = other;
            if (two.plan.order.by_group) two.plan = reordered(other.plan, perm);
        };
        consider(natural, 100);
        if (spill && two.plan.order.groups > 0) consider(joined, 103);
    }
    const bool on_pairs = two.plan.order.groups > 0;
    const int width = run.width;
    run.fill(plan, list);
    CUtensorMap mah, mal, mw[6];
    int rc = on_pairs ? FCB200_OK : map_half(&mah, a_hi, m, a_cols, lda, BM);
    if (!rc && !on_pairs) rc = map_half(&mal, a_lo, m, a_cols, lda, BM);
    int first = -1;
    for (int i = 0; i < 3 && !rc; ++i) {
        if (!used[i]) continue;
        if (first < 0) first = i;
        if (w_cols[i] % 8 || !aligned16(w_hi[i]) || !aligned16(w_lo[i]) || !(w_scale[i] > 0.f)) return FCB200_EINVAL;
        if (!on_pairs) rc = map_half(&mw[2 * i], w_hi[i], w_rows[i], w_cols[i], w_cols[i], width);
        if (!rc && !on_pairs) rc = map_half(&mw[2 * i + 1], w_lo[i], w_rows[i], w_cols[i], w_cols[i], width);
        prm.w_scale[i] = w_scale[i];
        prm.bias[i] = bias ? bias[i] : nullptr;
        if (prm.bias[i] && (!aligned16(prm.bias[i]) || w_rows[i] % BN)) return FCB200_EALIGN;
    }
    if (rc) return rc;
    for (int i = 0; i < 3; ++i)
        if (!used[i]) {  // never dereferenced; keep the parameter block initialised
            mw[2 * i] = mw[2 * first], mw[2 * i + 1] = mw[2 * first + 1];
            prm.w_scale[i] = 1.f;
        }
    if (ldy > 32767 || ldo > 32767) return FCB200_ERANGE;
    prm.y = y, prm.ldy = (int32_t)ldy, prm.y_cols = (int32_t)y_cols, prm.a_scale = a_scale, prm.o_scale = o_scale;
    prm.o_hi = static_cast<__half*>(o_hi), prm.o_lo = static_cast<__half*>(o_lo), prm.ldo = (int32_t)ldo;
    prm.rows_hi = rows_hi, prm.rows_lo = rows_lo, prm.ld_rows = (int32_t)ld_rows;
    prm.m_total = m, prm.status = status;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (on_pairs) return launch_pair(two.plan, prm, a_hi, a_lo, lda, a_cols, w_hi, w_lo, w_rows, w_cols, used, o_cols, forward, st);
    const int64_t items = plan.order.rows * plan.order.groups;
    const int grid = (int)(items < sm_count() ? items : sm_count());
    auto launch = [&](auto kind, auto columns) {
        constexpr int KIND = decltype(kind)::value, NB = decltype(columns)::value, bytes = kSmemBytes<NB>;
        static bool done[64] = {};
        const auto kernel = so2_conv_fused_kernel<KIND, NB>;
        if (const int arc = ensure_dynamic_smem(kernel, bytes, done)) return arc;
        launch_pdl(kernel, dim3(grid), dim3(kThreads), bytes, st, mah, mal, mw[0], mw[1], mw[2], mw[3], mw[4], mw[5], plan, prm);
        return launch_status();
    };
    auto by_width = [&](auto kind) {
        if (width == 32) return launch(kind, std::integral_constant<int, 32>{});
        if (width == 64) return launch(kind, std::integral_constant<int, 64>{});
        return launch(kind, std::integral_constant<int, 128>{});
    };
    if (forward) return by_width(std::integral_constant<int, kForwardKind>{});
    if (backward && rows_hi) return by_width(std::integral_constant<int, kPlanesKind>{});
    if (backward) return by_width(std::integral_constant<int, kBackwardKind>{});
    return by_width(std::integral_constant<int, kPlainKind>{});
}

}  // namespace fcb200

extern "C" int fcb200_so2_conv_fused(const void* a_hi, const void* a_lo, int64_t lda, int64_t a_cols, const void* const* w_hi,
                                     const void* const* w_lo, const int64_t* w_rows, const int64_t* w_cols,
                                     const float* w_scale, const float* const* bias, const int32_t* tiles, int32_t num_tiles,
                                     int32_t rot_begin, float* y, int64_t ldy, int64_t y_cols, void* o_hi, void* o_lo, int64_t ldo, int64_t o_cols,
                                     const float* a_scale, const float* o_scale, int64_t m, int32_t variant, int32_t* status,
                                     void* stream) {
    return so2_conv_fused(a_hi, a_lo, lda, a_cols, w_hi, w_lo, w_rows, w_cols, w_scale, bias, tiles, num_tiles, rot_begin, y, ldy, y_cols, o_hi, o_lo, ldo,
                          o_cols, a_scale, o_scale, m, variant, status, stream, nullptr, nullptr, 0);
}
