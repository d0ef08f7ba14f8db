// What the kernels of the SO(2) convolutions share (so2_conv_fused.cu: one CTA a row tile; so2_conv_pair.cu: two): tile
// lists, operand stages, packed float32 arithmetic and the half split.
#pragma once

#include "gemm_f16_common.cuh"

namespace fcb200 {
namespace fused {

using namespace f16;

enum Mode : int32_t {
    kPlain = 0,     // float32 tile -> y[:, out_col ...]; 1 is not assigned
    kSilu = 2,      // planes[:, out_col ...] = split(v * sigmoid(v));                       keep: y[:, y_col ...] = v
    kGated = 3,     // planes[:, out_col ...] = split(v * sigmoid(gate));                    keep: y[:, y_col ...] = v
    kSiluBwd = 4,   // planes[:, out_col ...] = split(v * d/dy silu(y[:, y_col ...]))
    kGatedBwd = 5,  // planes[:, out_col ...] = split(v * sigmoid(gate)); gate gradient summed over consecutive tiles
};
// kGateSilu: the gate is sigmoid(silu(g)), the scalar MLP of the node-wise feed-forward, instead of sigmoid(g).
// kGateSrc (set on the host): a gate tile of the rows that follow.
enum Flags : int32_t { kFirst = 1, kLast = 2, kKeep = 4, kGateSilu = 8, kGateSrc = 16 };

struct Tile {
    int16_t a_col;     // first input column of this tile's K range
    int16_t k;         // K extent (multiple of 32)
    int16_t w;         // weight matrix 0..2
    int16_t w_row;     // first output row of the weight matrix (multiple of 128)
    int16_t out_col;   // where the result goes (column of y for float32 modes, of the planes for split modes)
    int16_t mode;
    int16_t y_col;     // column of y holding this row's raw value (kSilu/kGated keep, kSiluBwd/kGatedBwd read)
    int16_t gate_col;  // column of y (and of the gradient planes) of the gate scalars of this row's degree
    int16_t flags;
};
constexpr int kMaxTiles = 40;   // tiles a caller may list; lmax 4: 19 rows x 2C = 38 column tiles in the conv-1 backward
constexpr int kMaxPlan = 80;    // tiles of a plan: a gate tile may be repeated for each of its rows

// What the epilogue of a launch has to be able to do; fixes how many registers it keeps between tiles.
// kPlanesKind: the gate's backward from the gated rows' own planes (see Params::rows_hi).
enum Kind { kPlainKind = 0, kForwardKind = 1, kBackwardKind = 2, kPlanesKind = 3 };

constexpr int KB = 64;               // k extent of a ring stage: 128-byte rows, 128-byte swizzle
constexpr int kPart = BM * KB * 2;   // 128 rows of one half plane of a stage, 16 KiB

// K-major, 128-byte swizzle: rows at a 128 B pitch, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t smem_desc128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;  // SWIZZLE_128B
    return d;
}

struct Params {
    const float* bias[3];
    float w_scale[3];
    float* y;          // raw conv-1 output / float32 output
    int32_t ldy, y_cols;
    __half *o_hi, *o_lo;
    int32_t ldo;
    const float* a_scale;  // power of two the A planes were written with (null = 1)
    const float* o_scale;  // power of two the output planes are written with (null = 1)
    // kPlanesKind: a gated row's gate gradient is made from what the forward pass gave the second convolution, a = y sigmoid(g),
    // instead of y: sum x y sigmoid'(g) = (1 - sigmoid(g)) sum x a.  Tile::y_col is a column of these planes.  a has 22 bits, below
    // 6e-5 (high half subnormal) an absolute error of 1.5e-11: a nearly closed gate's gradient is exact to that times sum |x|, no closer.
    const __half *rows_hi, *rows_lo;
    int32_t ld_rows;
    int64_t m_total;
    int32_t* status;
};

// Work items are row tiles times groups of tiles; `units` CTAs or pairs take them in turn, to and fro, either row by row (those
// that run together share an A tile in L2; to and fro, no unit is left with the costlier of two groups) or, by_group, group by
// group with the costly groups first, which leaves the last wave short where there are few items.
struct Order {
    int64_t rows;
    int32_t groups, by_group;
    // n-th item of a unit: its row tile and group; false past the last
    __host__ __device__ bool item(int64_t n, int64_t units, int64_t unit, int64_t& row, int& group) const {
        const int64_t i = n * units + (n & 1 ? units - 1 - unit : unit);
        if (i >= rows * groups) return false;
        if (by_group) {
            group = (int)(i / rows);
            row = i - group * rows;
        } else {
            row = i / groups;
            group = (int)(i - row * groups);
        }
        return true;
    }
};

// Tile list of a launch on CTA pairs: one or two listed tiles that read the same input columns.  A group is
// [begin[g], begin[g + 1]).
struct PairTile {
    int16_t a_col, k, w, n;  // n: listed tiles, 1 or 2
    int16_t w_row[2], out_col[2], mode[2], y_col[2], flags[2];
};
struct PairPlan {
    Order order;
    int16_t begin[kMaxTiles + 1];
    PairTile t[kMaxTiles];
};
int launch_pair(const PairPlan& plan, const Params& prm, const void* a_hi, const void* a_lo, int64_t lda, int64_t a_cols, const void* const* w_hi,
                const void* const* w_lo, const int64_t* w_rows, const int64_t* w_cols, const bool (&used)[3], int64_t o_cols, bool forward, cudaStream_t st);

// 1 / (1 + e^-v) on the special-function unit (ex2.approx, rcp.approx): relative error ~2^-22, a few instructions
// instead of the ~20 of expf and an IEEE division -- the epilogue evaluates it for every output element
__device__ __forceinline__ float sigmoid_f(float v) { return __fdividef(1.0f, 1.0f + __expf(-v)); }

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}
// D[tmem] (+)= A x B^T, issued by one lane of a warp in which every operand is the same in all lanes.
template <int N, bool kAdd>
__device__ __forceinline__ void umma_one(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
    if constexpr (kAdd)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "l"(da), "l"(db), "r"(instr_desc(N)) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "l"(da), "l"(db), "r"(instr_desc(N)), "r"(accumulate) : "memory");
}
// The warp waits as one, so that everything its loops derive from is the same in all lanes.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(kFull, mbar_wait(bar, parity, abort_flag));
}
// What a tensor map says, on its way before the first copy needs it.
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Two float32 in a register pair; the packed instructions halve the epilogue's multiply and add count.
typedef uint64_t f32x2;
__device__ __forceinline__ f32x2 pack(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
template <class F> __device__ __forceinline__ f32x2 map2(f32x2 v, F f) {
    float a, b;
    unpack(v, a, b);
    return pack(f(a), f(b));
}

// Two values -> packed halves hi and lo.  `top`: largest |hi| so far, NaN-propagating: an overflowed or invalid value
// becomes inf or NaN as a half, so one packed maximum per pair replaces range checks on the float32 values.
__device__ __forceinline__ void split2(f32x2 v, uint32_t& hi, uint32_t& lo, __half2& top) {
    float a, b;
    unpack(v, a, b);
    const __half2 h = __floats2half2_rn(a, b);
    const float2 hf = __half22float2(h);
    unpack(mul2(fma2(pack(hf.x, hf.y), pack(-1.f, -1.f), v), pack(kLoScale, kLoScale)), a, b);
    const __half2 l = __floats2half2_rn(a, b);
    top = __hmax2_nan(top, __habs2(h));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// hi and lo halves of four values -> the values
__device__ __forceinline__ void join2(uint64_t hi, uint64_t lo, f32x2& a, f32x2& b) {
    const uint32_t h[2] = {(uint32_t)hi, (uint32_t)(hi >> 32)}, l[2] = {(uint32_t)lo, (uint32_t)(lo >> 32)};
    const f32x2 s = pack(1.0f / kLoScale, 1.0f / kLoScale);
    auto wide = [](uint32_t v) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
        return pack(f.x, f.y);
    };
    a = fma2(wide(l[0]), s, wide(h[0])), b = fma2(wide(l[1]), s, wide(h[1]));
}

#define FCB_TMEM_LD16(r, taddr)                                                                                           \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "                                                                \
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"                         \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),        \
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])   \
                 : "r"(taddr)                                                                                             \
                 : "memory")

}  // namespace fused
}  // namespace fcb200
