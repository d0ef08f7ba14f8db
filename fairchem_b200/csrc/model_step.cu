// Host side of the whole-model evaluation: every launch of the forward and the backward pass from one call.
//
// Issued from Python, a launch costs 15-25 us of argument checks, views and allocations; with ~650 of them an evaluation
// took 16-18 ms however small the system was (21 atoms: 4.4 ms of kernel time in 16 ms).  Here a launch costs what the
// runtime needs, buffers come from two caller-owned blocks by adding offsets, and what used to be separate launches is
// grouped: the hidden layers of all radial MLPs run side by side, the nine (25) per-row linears of the node feed-forward
// are one launch with the gate in its epilogue, residual adds live in the norm and rotate-back kernels.
#include "edge_step.cuh"
#include "node_step.cuh"

#include <vector>

#include "gemm_common.cuh"

namespace fcb200 {
namespace step {

static fcb200_launch_hook g_hook = nullptr;

#define FCB_TRY(expr)                    \
    do {                                 \
        const int rc_ = (expr);          \
        if (rc_ != FCB200_OK) return rc_; \
    } while (0)

struct Arena {
    char* base;
    int64_t off = 0;
    template <class T> T* take(int64_t count) {
        T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
        off += (count * (int64_t)sizeof(T) + 1023) / 1024 * 1024;
        return p;
    }
};

struct Planes {
    __half *hi = nullptr, *lo = nullptr;
    int64_t ld = 0;  // elements per row
    OutSplit out() const { return OutSplit{hi, lo, 1.0f}; }
    Planes from(int64_t row) const {
        Planes p = *this;
        p.hi += row * ld, p.lo += row * ld;
        return p;
    }
};

// sizes that follow from lmax
struct Dims {
    int lmax, nl, nm, nw, nrad, gates, yw, kw;  // yw: conv 1's columns, kw: of those, gates and row 0
    explicit Dims(int l) : lmax(l), nl((l + 1) * (l + 1)), nm((l + 1) + 2 * l + 2 * (l - 1)), nw(l == 2 ? Shape<2>::kW : Shape<4>::kW),
                           nrad(3 * l), gates(l * C), yw((l + nm) * C), kw((l + 1) * C) {}
};

struct Layer {
    float *x0, *xn1, *st1, *x1, *st2, *ffn_y;  // inputs of the two norms, first norm's output, feed-forward pre-activation
    float *y, *msg, *rad;                      // conv-1 output, messages, radial weights (per edge); null: not kept
    // Where everything fits, the gated rows are kept for the backward pass as conv 2 read them, and of the conv-1 output only
    // the gates and row 0: one row more to keep, but eight (lmax 4: 18) of 4 bytes fewer to write.  Forces then differ by some 2e-7 from
    // those of the smaller kept sets, whose gate gradients are made from float32 rows and which agree bit for bit among themselves.
    Planes a;
    int64_t yw = 0;                            // columns of y
};

struct Layout {
    int64_t n, e, ec;
    int nets;
    int64_t rw;  // width of the radial hidden tensors
    // kept from forward to backward
    float4* vec;
    float *wig, *env, *sys, *pre1, *pre2, *rst1, *rst2, *xl, *stl, *hy1, *hy2;
    __half* h2;  // [E, nets, 2, C]: hi | lo of the second hidden activation; the backward pass reuses it as float [E, nets*C]
    Planes row0, hh;
    std::vector<Layer> layer;
    int64_t keep_bytes;
    // forward scratch
    Planes gauss, h1, m, a, xn2, a2;
    float *radial, *ffn_out, *r3, *y_c, *msg_c;
    // backward scratch
    Planes gp, gy2, gmsg, gy, grad, gr3, rp, hg;
    float *g, *g1, *gxn, *gm, *rh, *ggauss, *grad_vec, *tau_n, *tau_e, *g0, *rad_scale;
    Scale* scales;
    int64_t scratch_bytes;
};

static Planes planes(Arena& a, int64_t rows, int64_t width) {
    Planes p;
    p.hi = a.take<__half>(rows * width);
    p.lo = a.take<__half>(rows * width);
    p.ld = width;
    return p;
}

// backward: which pass owns the scratch block (the two passes share its memory, and the tensors both need are placed per pass)
static void lay_out(const fcb200_model& md, const fcb200_eval& ev, bool backward, Layout& L) {
    const Dims d(md.lmax);
    const int64_t n = L.n = ev.num_nodes, e = L.e = ev.num_edges;
    L.ec = 0;
    for (int c = 0; c < ev.num_chunks; ++c) L.ec = std::max(L.ec, ev.chunk_edge[c + 1] - ev.chunk_edge[c]);
    const int64_t ec = L.ec;
    L.nets = md.num_layers + 1;
    L.rw = (int64_t)L.nets * C;
    const bool keep = ev.want_grad != 0, planes_kept = ev.keep_radial == 1;
    // per-edge tensors that only the backward pass reads shrink to one chunk when there is none; row counts of the large
    // ones are rounded up so that a slowly changing edge count (molecular dynamics) asks for the same block every step
    int64_t unit = 1024;  // 1/64 to 1/32 of the edges
    while (unit * 64 < e) unit *= 2;
    const int64_t er = (e + unit - 1) / unit * unit, ek = keep ? er : ec;
    Arena k{static_cast<char*>(ev.keep)};
    L.vec = k.take<float4>(er);
    L.wig = k.take<float>(er * d.nw);
    L.env = k.take<float>(er);
    L.sys = k.take<float>((int64_t)ev.num_systems * C);
    L.pre1 = k.take<float>(ek * L.rw);
    L.pre2 = k.take<float>(ek * L.rw);
    L.rst1 = k.take<float>(ek * L.nets * 2);
    L.rst2 = k.take<float>(ek * L.nets * 2);
    L.h2 = k.take<__half>(er * L.rw * 2);
    L.xl = k.take<float>(n * d.nl * C);
    L.stl = k.take<float>(n * 2);
    L.hy1 = k.take<float>(n * C);
    L.hy2 = k.take<float>(n * C);
    L.row0 = planes(k, n, C);
    L.hh = planes(k, n, C);
    L.layer.resize(md.num_layers);
    for (int l = 0; l < md.num_layers; ++l) {
        Layer& q = L.layer[l];
        if (l > 0 && !keep) {  // nothing is read again: all layers share one set
            q = L.layer[0];
            continue;
        }
        q.x0 = k.take<float>(n * d.nl * C);
        q.xn1 = k.take<float>(n * d.nl * C);
        q.st1 = k.take<float>(n * 2);
        q.x1 = k.take<float>(n * d.nl * C);
        q.st2 = k.take<float>(n * 2);
        q.ffn_y = k.take<float>(n * (md.lmax + d.nl) * C);
        const bool edges = keep && l >= ev.drop_layers;
        q.yw = planes_kept ? d.kw : d.yw;
        q.y = edges ? k.take<float>(er * q.yw) : nullptr;
        q.a = edges && planes_kept ? planes(k, er, d.nm * C) : Planes{};
        q.msg = edges ? k.take<float>(er * d.nm * C) : nullptr;
        q.rad = edges && ev.keep_radial ? k.take<float>(er * d.nrad * 2 * C) : nullptr;
    }
    L.keep_bytes = k.off;

    Arena b{static_cast<char*>(ev.scratch)};
    if (!backward) {
        L.gauss = planes(b, e, md.num_basis);
        L.h1 = planes(b, ec, L.rw);
        L.r3 = b.take<float>(ec * (md.lmax + 1) * C);
        L.radial = b.take<float>(ec * d.nrad * 2 * C);
        L.m = planes(b, ec, d.nm * 2 * C);
        const bool all = keep && ev.drop_layers <= 0;
        if (!all || !planes_kept) L.a = planes(b, ec, d.nm * C);
        L.y_c = all ? nullptr : b.take<float>(ec * d.gates);
        L.msg_c = all ? nullptr : b.take<float>(ec * d.nm * C);
        L.xn2 = planes(b, n, d.nl * C);
        L.a2 = planes(b, n, d.nl * C);
        L.ffn_out = b.take<float>(n * d.nl * C);
        L.scratch_bytes = b.off;
        return;
    }
    L.scales = b.take<Scale>(2 * md.num_layers + 1);
    L.rad_scale = b.take<float>(1);
    L.g = b.take<float>(n * d.nl * C);
    L.g1 = b.take<float>(n * d.nl * C);
    L.gxn = b.take<float>(n * d.nl * C);
    L.g0 = b.take<float>(n * C);
    L.hg = planes(b, n, C);
    L.gp = planes(b, n, d.nl * C);
    L.gy2 = planes(b, n, (md.lmax + d.nl) * C);
    L.tau_n = b.take<float>(e * 4);
    L.tau_e = b.take<float>(e * 4);
    L.grad_vec = b.take<float>(e * 3);
    const int64_t edge_part = b.off;
    // the layers
    L.radial = b.take<float>(ec * d.nrad * 2 * C);
    L.gmsg = planes(b, ec, d.nm * C);
    L.gy = planes(b, ec, d.yw);
    L.gm = b.take<float>(ec * d.nm * 2 * C);
    L.grad = planes(b, ec, d.nrad * 2 * C);
    const int64_t layers_end = b.off;
    // A layer that keeps nothing per edge is computed again on the memory of gradients that come later in its chunk:
    // the rotated rows where theirs go, the gated rows in the message gradient, the messages and the conv-1 output in the
    // planes of the conv-1 output's and the radial weights' gradients (4 bytes an element each, like float32).
    L.m.hi = reinterpret_cast<__half*>(L.gm), L.m.lo = L.m.hi + ec * d.nm * 2 * C, L.m.ld = d.nm * 2 * C;
    L.a = L.gmsg;
    L.msg_c = reinterpret_cast<float*>(L.gy.hi);
    L.y_c = reinterpret_cast<float*>(L.grad.hi);
    static_assert(2 + 9 <= 6 * 2 && 4 + 19 <= 12 * 2, "yw fits the radial gradient of lmax 2 and 4");
    b.off = edge_part;  // the radial MLPs' backward runs after the layers, on the same memory
    L.r3 = b.take<float>(ec * (md.lmax + 1) * C);
    L.gr3 = planes(b, ec, (md.lmax + 1) * C);
    L.rp = planes(b, ec, L.rw);
    L.rh = b.take<float>(ec * L.rw);
    L.ggauss = b.take<float>(ec * md.num_basis);
    L.scratch_bytes = std::max(layers_end, b.off);
}

// ---- contractions ------------------------------------------------------------------------------------------------
constexpr int kPlain = 0, kSilu = 2, kGated = 3, kSiluBwd = 4, kGatedBwd = 5;
constexpr int kFirst = 1, kLast = 2, kKeep = 4, kGateSilu = 8;

struct Conv {
    std::vector<int32_t> t;
    const fcb200_weight* w[3] = {};
    const float* bias[3] = {};
    int64_t macs = 0;
    void tile(int a_col, int k, int wi, int w_row, int out_col, int mode = kPlain, int y_col = 0, int gate_col = 0, int flags = 0) {
        const int v[9] = {a_col, k, wi, w_row, out_col, mode, y_col, gate_col, flags};
        t.insert(t.end(), v, v + 9);
        macs += 128LL * k;
    }
    int count() const { return (int)t.size() / 9; }
};

struct Run {
    const fcb200_model& md;
    const fcb200_eval& ev;
    Dims d;
    Layout L;
    cudaStream_t st;
    void* stream;
    Run(const fcb200_model& m, const fcb200_eval& e, void* s, bool backward) : md(m), ev(e), d(m.lmax), st(static_cast<cudaStream_t>(s)), stream(s) {
        lay_out(m, e, backward, L);
        pdl_launches = e.num_edges <= kPdlEdges;
    }
    ~Run() { pdl_launches = false; }
    Run(const Run&) = delete;

    void hook(const char* name, int begin, int64_t bytes, int64_t flops = 0, int launches = 1) const {
        if (g_hook) g_hook(name, begin, bytes, flops, launches);
    }
    // f() launches the kernel(s) of one step
    template <class F> int op(const char* name, int64_t bytes, F&& f, int64_t flops = 0, int launches = 1) const {
        hook(name, 1, bytes, flops, launches);
        int rc = f();
        if (rc == FCB200_OK) rc = launch_status();
        hook(name, 0, bytes, flops, launches);
        return rc;
    }

    // one launch of tile list c on rows [m] of half planes
    int conv(const char* name, const Conv& c, const void* a_hi, const void* a_lo, int64_t lda, int64_t a_cols, int rot_begin, float* y,
             int64_t ldy, int64_t y_cols, const Planes* o, int64_t o_cols, const float* a_scale, const float* o_scale, int64_t m, const Planes* gated = nullptr) const {
        const void *hi[3] = {}, *lo[3] = {};
        int64_t rows[3] = {}, cols[3] = {};
        float sc[3] = {1.f, 1.f, 1.f};
        for (int i = 0; i < 3; ++i)
            if (c.w[i]) hi[i] = c.w[i]->hi, lo[i] = c.w[i]->lo, rows[i] = c.w[i]->rows, cols[i] = c.w[i]->cols, sc[i] = c.w[i]->scale;
        const int64_t bytes = 4 * m * (a_cols + 128LL * c.count()), flops = 2 * m * c.macs;
        hook(name, 1, bytes, flops);
        const int rc = so2_conv_fused(a_hi, a_lo, lda, a_cols, hi, lo, rows, cols, sc, c.bias, c.t.data(), c.count(), rot_begin, y,
                                             ldy, y_cols, o ? o->hi : nullptr, o ? o->lo : nullptr, o ? o->ld : 0, o_cols, a_scale,
                                             o_scale, m, 0, ev.status, stream, gated ? gated->hi : nullptr, gated ? gated->lo : nullptr, gated ? gated->ld : 0);
        hook(name, 0, bytes, flops);
        return rc;
    }
    // c [m, w.rows] = planes x w^T
    int gemm(const char* name, const Planes& a, const fcb200_weight& w, const float* scale, float* c, int64_t ldc, int64_t m) const {
        return conv(name, linear(w, nullptr), a.hi, a.lo, a.ld, w.cols, 0, c, ldc, w.rows, nullptr, 0, scale, nullptr, m);
    }

    // plain tiles of the m-blocks w[0..2] side by side (transposed = the given matrices are already the transposes)
    static Conv blocks(const fcb200_weight* w) {
        Conv c;
        int a = 0, o = 0;
        for (int i = 0; i < 3; ++i) {
            c.w[i] = w + i;
            for (int r = 0; r < w[i].rows; r += C) c.tile(a, w[i].cols, i, r, o + r);
            a += w[i].cols, o += w[i].rows;
        }
        return c;
    }
    static Conv linear(const fcb200_weight& w, const float* bias) {
        Conv c;
        c.w[0] = &w, c.bias[0] = bias;
        for (int r = 0; r < w.rows; r += C) c.tile(0, w.cols, 0, r, r);
        return c;
    }
    int degree_of_row(int r) const {  // M-major row -> degree
        if (r <= d.lmax) return r;
        r -= d.lmax + 1;
        if (r < 2 * d.lmax) return r % d.lmax + 1;
        return (r - 2 * d.lmax) % (d.lmax - 1) + 2;
    }
    enum Keep { kNothing, kRow0, kRows };  // which of conv 1's raw rows go to y
    Conv conv1_gate(int l, Keep keep) const;
    int messages(int l, const Conv& c1, int64_t e0, int64_t ec, float* y, int64_t yw, float* msg) const;
    int forward();
    int energy();
    int backward();
    int radial_hidden_forward();
    int layer_forward(int l, const float* ffn_prev);
    int ffn_forward(int l);
    int layer_backward(int l);

    const float* radial_of(int l, int64_t e0) const { return L.layer[l].rad ? L.layer[l].rad + e0 * d.nrad * 2 * C : L.radial; }
    int radial_out(int l, int64_t e0, int64_t ec) const {
        const __half* h = L.h2 + e0 * L.rw * 2 + (int64_t)l * 2 * C;
        return conv("so2_conv_fused_radial_out", linear(md.layers[l].radial_out, md.layers[l].radial_out_bias), h, h + C, L.rw * 2, C, 0,
                    const_cast<float*>(radial_of(l, e0)), d.nrad * 2 * C, d.nrad * 2 * C, nullptr, 0, nullptr, nullptr, ec);
    }
    int degree_out(int64_t e0, int64_t ec) const {
        const __half* h = L.h2 + e0 * L.rw * 2 + (int64_t)md.num_layers * 2 * C;
        return conv("so2_conv_fused_radial_out", linear(md.degree_out, md.degree_out_bias), h, h + C, L.rw * 2, C, 0, L.r3,
                    (d.lmax + 1) * C, (d.lmax + 1) * C, nullptr, 0, nullptr, nullptr, ec);
    }
    template <class F> int chunks(F&& f) const {
        for (int c = 0; c < ev.num_chunks; ++c) FCB_TRY(f(c, ev.chunk_edge[c], ev.chunk_edge[c + 1] - ev.chunk_edge[c], ev.chunk_node[c], ev.chunk_node[c + 1]));
        return FCB200_OK;
    }
    template <class F> int by_lmax(F&& f) const {
        return d.lmax == 2 ? f(std::integral_constant<int, 2>{}) : f(std::integral_constant<int, 4>{});
    }
    BasisParams basis() const { return make_basis(md.cutoff, md.num_basis, md.basis_start, md.basis_stop, md.basis_width); }
    const int32_t* src_lo(int c) const { return ev.num_chunks > 1 ? ev.chunk_src + (int64_t)c * L.n : ev.src_ptr; }
    const int32_t* src_hi(int c) const { return ev.num_chunks > 1 ? ev.chunk_src + (int64_t)(c + 1) * L.n : ev.src_ptr + 1; }
};

// Kernels that walk a node's edges: with one warp per node, few nodes leave warp slots of the 148 SMs idle while each
// walks ~30 edges in turn, so a block of several warps shares the node's edges.  From about 12 warps per SM (what the
// registers of the backward gather allow) on, one warp per node is the faster form (2000 nodes: 1.42 ms shared, 1.30
// alone per four layers; 256 nodes: 0.23 against 0.88).
static bool share_node(int64_t nodes) { return nodes < 148 * 8; }

template <class K> static int raise_smem(K kernel, int bytes, bool (&done)[64]) { return bytes > 48 * 1024 ? ensure_dynamic_smem(kernel, bytes, done) : FCB200_OK; }

template <int LMAX, int MODE>
static int launch_rotate_back(const Run& r, const float* msg, int64_t e_base, const float* residual, float* out, int64_t n0, int64_t n1) {
    const fcb200_eval& ev = r.ev;
    const float inv = MODE == 1 ? 1.0f / r.md.rescale : 1.0f;
    auto shared = [&](auto tag) {
        constexpr int WPN = decltype(tag)::value, bytes = WPN * Shape<LMAX>::kL * C * 4;
        static bool done[64] = {};
        FCB_TRY(raise_smem(rotate_back_kernel<LMAX, MODE, WPN>, bytes, done));
        launch_pdl((rotate_back_kernel<LMAX, MODE, WPN>), dim3((int)(n1 - n0)), dim3(WPN * 32), bytes, r.st, msg, r.L.wig, r.L.env, ev.row_ptr, e_base, residual, r.md.element_emb, ev.z, r.L.sys, ev.batch, out, inv, n0, n1);
        return (int)FCB200_OK;
    };
    // Eight warps to a node, or four where those take less in all at lmax 4: one block of eight fills an SM's registers and lasts 0.63
    // times as long as one of four, of which two fit.  us a launch, 8 / 4 warps, by nodes: 108 14.8 / 18.8, 256 28.7 / 26.6, 400 42.8 / 47.0,
    // 576 58.8 / 53.4, 864 80.1 / 75.3, 1 176 109 / 99; lmax 2, 256 12.6 / 14.7, 720 31.1 / 31.5.  Off by little, and left so because the number of
    // warps is the order of a node's sum: lmax 4, 720 nodes 69.9 / 71.7; the m = 0 rows alone (three blocks of four fit), 400 nodes
    // 23.6 / 16.9 once an evaluation of 15.6 ms; lmax 2, 400 nodes 18.7 / 16.7.
    const int64_t n = n1 - n0, sms = sm_count(), rounds = (n + sms - 1) / sms, halves = (n + 2 * sms - 1) / (2 * sms);
    if (share_node(n)) {
        if constexpr (LMAX == 4)
            if (63 * rounds >= 100 * halves) return shared(std::integral_constant<int, 4>{});
        return shared(std::integral_constant<int, 8>{});
    } else {
        launch_pdl((rotate_back_kernel<LMAX, MODE, 1>), dim3(warp_grid(n1 - n0, 4)), dim3(128), 0, r.st, msg, r.L.wig, r.L.env, ev.row_ptr, e_base, residual, r.md.element_emb, ev.z, r.L.sys, ev.batch, out, inv, n0, n1);
    }
    return FCB200_OK;
}

template <int LMAX, int HALF>
static int launch_gather_bwd(const Run& r, const float* x, const int32_t* lo, const int32_t* hi, const float* radial, float* gx, bool store_gx, bool store_tau,
                             const float* scale, int64_t e0, int64_t n0, int64_t n1) {
    const Layout& L = r.L;
    constexpr int bytes = 2 * kGatherRows * C * 4, alone = ahead<LMAX, HALF> ? 4 * bytes : 0;  // of a warp, of a block of four nodes
    static bool done[3][64] = {};
    auto shared = [&](auto tag, bool (&up)[64]) {
        constexpr int WPN = decltype(tag)::value;
        FCB_TRY(raise_smem(gather_bwd_kernel<LMAX, HALF, WPN, OutSplit>, WPN * bytes, up));
        launch_pdl((gather_bwd_kernel<LMAX, HALF, WPN, OutSplit>), dim3((int)(n1 - n0)), dim3(WPN * 32), WPN * bytes, r.st, L.gm, x, lo, hi, r.ev.src_perm, L.wig, radial, gx, (int)store_gx, L.tau_n, (int)store_tau, L.grad.out(), scale, e0, n0, n1);
        return (int)FCB200_OK;
    };
    // Twelve warps fit an SM.  Four to a node where whole waves of one node a warp would leave the last one nearly empty
    // (us of an evaluation, lmax 2: 1 296 nodes 688 -> 656, 1 782 1026 -> 904, 2 000 1198 -> 1002, 2 592 1384 -> 1259, 4 050 2076 ->
    // 1951; where it does not: 1 440 731 -> 771, 3 120 1496 -> 1529, 5 280 2414 -> 2545; lmax 4, 2 048 nodes 9662 -> 7773).
    // More nodes come in several chunks, which hold too few edges of a source to share.
    // Fewer nodes: eight warps to a node, one block on an SM, unless four and three blocks take fewer rounds; a round of those
    // lasts 2.05 times as long (us a launch, mean of by source and by target, 8 / 4 warps, by nodes: 144 15.5 / 19.7, 432 39.6 / 32.8,
    // 720 60.5 / 53.6, 1 176 94 / 81; lmax 4, 144 41 / 55, 256 61 / 65, 432 94 / 84, 500 117 / 129, 720 161 / 148, 1 176 270 / 230).  At lmax 2 the ratio is
    // just below 2 (256 nodes 27.2 / 26.2, 500 nodes 46.9 / 45.2); left so because the number of warps is the order of a node's sum.
    const int64_t n = n1 - n0, sms = sm_count(), waves = (n + 12 * sms - 1) / (12 * sms), quarters = (n + 3 * sms - 1) / (3 * sms), rounds = (n + sms - 1) / sms;
    if (share_node(n) && 20 * rounds <= 41 * quarters) {
        FCB_TRY(shared(std::integral_constant<int, 8>{}, done[0]));
    } else if (share_node(n) || (waves <= 3 && 11 * quarters < 40 * waves)) {
        FCB_TRY(shared(std::integral_constant<int, 4>{}, done[2]));
    } else {
        FCB_TRY(raise_smem(gather_bwd_kernel<LMAX, HALF, 1, OutSplit>, alone, done[1]));
        launch_pdl((gather_bwd_kernel<LMAX, HALF, 1, OutSplit>), dim3(warp_grid(n1 - n0, 4)), dim3(128), alone, r.st, L.gm, x, lo, hi, r.ev.src_perm, L.wig, radial, gx, (int)store_gx, L.tau_n, (int)store_tau, L.grad.out(), scale, e0, n0, n1);
    }
    return FCB200_OK;
}

int Run::radial_hidden_forward() {
    const int nets = L.nets;
    Conv c0, c1;
    c0.w[0] = &md.rad_w0, c0.bias[0] = md.rad_b0;
    c1.w[0] = &md.rad_w1, c1.bias[0] = md.rad_b1;
    for (int i = 0; i < nets; ++i) {
        c0.tile(0, md.num_basis, 0, i * C, i * C);
        c1.tile(i * C, C, 0, i * C, i * C);
    }
    return chunks([&](int, int64_t e0, int64_t ec, int64_t, int64_t) {
        const int64_t k0 = ev.want_grad ? e0 : 0;
        float *pre1 = L.pre1 + k0 * L.rw, *pre2 = L.pre2 + k0 * L.rw;
        FCB_TRY(conv("so2_conv_fused_radial_in", c0, L.gauss.hi + e0 * md.num_basis, L.gauss.lo + e0 * md.num_basis, md.num_basis, md.num_basis,
                     0, pre1, L.rw, L.rw, nullptr, 0, nullptr, nullptr, ec));
        const int grid = warp_grid(radial_items(ec, nets, kRadialFwdRows), 8);
        FCB_TRY(op("radial_act_fwd", ec * nets * 1040, [&] {
            launch_pdl(radial_fwd_kernel, dim3(grid), dim3(256), 0, st, pre1, md.table_src, md.table_tgt, ev.z, ev.src + e0, ev.tgt + e0, md.ln1_w, md.ln1_b, md.radial_eps,
                                                    L.h1.out(), C, L.rst1 + k0 * nets * 2, ec * nets, nets);
            return 0;
        }));
        FCB_TRY(conv("so2_conv_fused_radial_in", c1, L.h1.hi, L.h1.lo, L.rw, L.rw, 0, pre2, L.rw, L.rw, nullptr, 0, nullptr, nullptr, ec));
        __half* h = L.h2 + e0 * L.rw * 2;
        return op("radial_act_fwd", ec * nets * 1032, [&] {
            launch_pdl(radial_fwd_kernel, dim3(grid), dim3(256), 0, st, pre2, nullptr, nullptr, ev.z, ev.src + e0, ev.tgt + e0, md.ln2_w, md.ln2_b, md.radial_eps,
                                                    OutSplit{h, h + C, 1.0f}, 2 * C, L.rst2 + k0 * nets * 2, ec * nets, nets);
            return 0;
        });
    });
}

// conv 1 with the gate in its epilogue: gate tiles first, then the rows
Conv Run::conv1_gate(int l, Keep keep) const {
    Conv c = blocks(md.layers[l].conv1);
    c.bias[0] = md.layers[l].conv1_bias;
    for (int i = d.lmax; i < c.count(); ++i) {
        int32_t* t = &c.t[9 * i];
        const int r = i - d.lmax;
        t[4] = r * C;
        t[5] = r == 0 ? kSilu : kGated;
        t[6] = (d.lmax + r) * C;
        t[7] = r == 0 ? 0 : (degree_of_row(r) - 1) * C;
        t[8] = keep == kRows || (keep == kRow0 && r == 0) ? kKeep : 0;
    }
    return c;
}

// messages of a chunk's edges: radial weights, gather + rotate, conv 1 + gate, conv 2; y [ec, yw] takes conv 1's raw values
int Run::messages(int l, const Conv& c1, int64_t e0, int64_t ec, float* y, int64_t yw, float* msg) const {
    const Layer& q = L.layer[l];
    FCB_TRY(radial_out(l, e0, ec));
    const int64_t gb = ec * (4LL * (2 * d.nl * C + 2 * d.nm * C + d.nw + d.nrad * 2 * C) + 8);
    FCB_TRY(op("gather_rotate_fwd", gb, [&] {
        return by_lmax([&](auto lm) {
            constexpr int LM = decltype(lm)::value;
            launch_pdl(gather_fwd_kernel<LM>, dim3(warp_grid(2 * ec, 4, 148 * (LM == 2 ? 5 : 3) * 4)), dim3(128), 0, st, q.xn1, ev.src + e0, ev.tgt + e0, L.wig + e0 * d.nw, radial_of(l, e0), L.m.out(), ec);
            return 0;
        });
    }));
    const Planes a = q.a.hi ? q.a.from(e0) : L.a;
    FCB_TRY(conv("so2_conv_fused_conv1_gate", c1, L.m.hi, L.m.lo, L.m.ld, L.m.ld, d.lmax, y, yw, yw, &a, a.ld, nullptr, nullptr, ec));
    Conv c2 = blocks(md.layers[l].conv2);
    c2.bias[0] = md.layers[l].conv2_bias;
    return conv("so2_conv_fused_conv2", c2, a.hi, a.lo, a.ld, a.ld, 0, msg, d.nm * C, d.nm * C, nullptr, 0, nullptr, nullptr, ec);
}

int Run::layer_forward(int l, const float* ffn_prev) {
    const fcb200_layer& w = md.layers[l];
    const Layer& q = L.layer[l];
    const int64_t n = L.n, row = d.nl * C;
    const float* x_prev = l == 0 ? q.x0 : L.layer[l - 1].x1;
    FCB_TRY(op("rms_norm_sh_fwd", n * row * 4 * (ffn_prev ? 4 : 2), [&] {
        return by_lmax([&](auto lm) {
            launch_pdl(norm_fwd_kernel<decltype(lm)::value>, dim3(warp_grid(n, 4)), dim3(128), 0, st, x_prev, ffn_prev, q.x0, w.norm1_w, w.norm1_b, L.sys, ev.batch,
                                                                                q.xn1, OutSplit{}, OutSplit{}, q.st1, w.eps1, n);
            return 0;
        });
    }));
    const Conv c1 = conv1_gate(l, q.a.hi ? kRow0 : q.y ? kRows : kNothing);
    return chunks([&](int, int64_t e0, int64_t ec, int64_t n0, int64_t n1) {
        float* msg = q.msg ? q.msg + e0 * d.nm * C : L.msg_c;
        FCB_TRY(messages(l, c1, e0, ec, q.y ? q.y + e0 * q.yw : L.y_c, q.y ? q.yw : d.gates, msg));
        return op("rotate_back_reduce_fwd", ec * 4 * (d.nm * C + d.nw) + (n1 - n0) * row * 8,
                  [&] { return by_lmax([&](auto lm) { return launch_rotate_back<decltype(lm)::value, 0>(*this, msg, e0, q.x0, q.x1, n0, n1); }); });
    });
}

int Run::ffn_forward(int l) {
    const fcb200_layer& w = md.layers[l];
    const Layer& q = L.layer[l];
    const int64_t n = L.n, row = d.nl * C;
    FCB_TRY(op("rms_norm_sh_fwd", n * row * 8, [&] {
        return by_lmax([&](auto lm) {
            launch_pdl(norm_fwd_kernel<decltype(lm)::value>, dim3(warp_grid(n, 4)), dim3(128), 0, st, q.x1, nullptr, nullptr, w.norm2_w, w.norm2_b, nullptr, nullptr,
                                                                                nullptr, L.xn2.out(), OutSplit{}, q.st2, w.eps2, n);
            return 0;
        });
    }));
    Conv c1, c2;
    c1.w[0] = &w.ffn_in, c1.bias[0] = w.ffn_in_bias;
    c2.w[0] = &w.ffn_out, c2.bias[0] = w.ffn_out_bias;
    for (int i = 0; i < d.lmax; ++i) c1.tile(0, C, 0, i * C, i * C);
    for (int r = 0; r < d.nl; ++r) {
        const int deg = degree_of(r);
        c1.tile(r * C, C, 0, (d.lmax + deg) * C, r * C, r == 0 ? kSilu : kGated, (d.lmax + r) * C, r == 0 ? 0 : (deg - 1) * C, kKeep | kGateSilu);
        c2.tile(r * C, C, 0, deg * C, r * C);
    }
    const int64_t yw = (d.lmax + d.nl) * C;
    FCB_TRY(conv("ffn_in_gate", c1, L.xn2.hi, L.xn2.lo, row, row, d.lmax, q.ffn_y, yw, yw, &L.a2, row, nullptr, nullptr, n));
    return conv("ffn_out", c2, L.a2.hi, L.a2.lo, row, row, 0, L.ffn_out, row, row, nullptr, 0, nullptr, nullptr, n);
}

int Run::forward() {
    const int64_t n = L.n, e = L.e;
    FCB_TRY(op("system_embedding", 0, [&] {
        launch_pdl(system_kernel, dim3(ev.num_systems), dim3(8 * C), 0, st, ev.charge, ev.spin, ev.dataset, md.charge_emb, md.spin_emb, md.dataset_emb, md.csd_w_t, md.csd_b,
                                                    L.sys, ev.status);
        return 0;
    }));
    FCB_TRY(op("edge_geometry_fwd", e * 4 * (5 + d.nw + md.num_basis + 8), [&] {
        return by_lmax([&](auto lm) {
            constexpr int LM = decltype(lm)::value;
            constexpr int bytes = 128 * Shape<LM>::kW * 4;
            static bool done[64] = {};
            FCB_TRY(raise_smem(geometry_fwd_kernel<LM>, bytes, done));
            launch_pdl(geometry_fwd_kernel<LM>, dim3((unsigned)((e + 127) / 128)), dim3(128), bytes, st, ev.pos, ev.src, ev.tgt, ev.shift, ev.gamma, L.vec, L.env, L.wig,
                                                                                    L.gauss.hi, L.gauss.lo, basis(), e);
            return 0;
        });
    }));
    FCB_TRY(radial_hidden_forward());
    FCB_TRY(chunks([&](int, int64_t e0, int64_t ec, int64_t n0, int64_t n1) {
        FCB_TRY(degree_out(e0, ec));
        return op("edge_degree_fwd", ec * 4 * ((d.lmax + 1) * C + d.nw) + (n1 - n0) * d.nl * C * 4, [&] {
            return by_lmax([&](auto lm) { return launch_rotate_back<decltype(lm)::value, 1>(*this, L.r3, e0, nullptr, L.layer[0].x0, n0, n1); });
        });
    }));
    for (int l = 0; l < md.num_layers; ++l) {
        FCB_TRY(layer_forward(l, l == 0 ? nullptr : L.ffn_out));
        FCB_TRY(ffn_forward(l));
    }
    return op("rms_norm_sh_fwd", n * d.nl * C * 16, [&] {
        return by_lmax([&](auto lm) {
            launch_pdl(norm_fwd_kernel<decltype(lm)::value>, dim3(warp_grid(n, 4)), dim3(128), 0, st, L.layer.back().x1, L.ffn_out, L.xl, md.norm_w, md.norm_b, nullptr,
                                                                                nullptr, ev.x_out, OutSplit{}, L.row0.out(), L.stl, md.norm_eps, n);
            return 0;
        });
    });
}

int Run::energy() {
    const int64_t n = L.n;
    Conv c1, c2;
    c1.w[0] = &md.head_w1, c1.bias[0] = md.head_b1;
    c2.w[0] = &md.head_w2, c2.bias[0] = md.head_b2;
    c1.tile(0, C, 0, 0, 0, kSilu, 0, 0, kKeep);
    c2.tile(0, C, 0, 0, 0);
    FCB_TRY(conv("head", c1, L.row0.hi, L.row0.lo, C, C, 0, L.hy1, C, C, &L.hh, C, nullptr, nullptr, n));
    FCB_TRY(conv("head", c2, L.hh.hi, L.hh.lo, C, C, 0, L.hy2, C, C, nullptr, 0, nullptr, nullptr, n));
    const int per = n < 148 * 64 ? 1 : 16;
    return op("energy_sum", n * C * 4, [&] {
        launch_pdl(energy_kernel, dim3((unsigned)((n + 8 * per - 1) / (8 * per))), dim3(256), 0, st, L.hy2, md.head_w3, md.head_b3, ev.batch, ev.energy, n, per);
        return 0;
    });
}

int Run::layer_backward(int l) {
    const fcb200_layer& w = md.layers[l];
    const Layer& q = L.layer[l];
    const int64_t n = L.n, row = d.nl * C;
    const int k = 2 * (md.num_layers - 1 - l);
    Scale* s = L.scales + k;
    // node feed-forward
    FCB_TRY(op("split_planes", n * row * 8, [&] { launch_pdl(split_kernel, dim3(warp_grid(n * row / 4, 256)), dim3(256), 0, st, L.g, L.gp.out(), &s->scale, n * row / 4); return 0; }));
    Conv b2, b1;
    b2.w[0] = &w.ffn_out_t;
    b1.w[0] = &w.ffn_in_t0, b1.w[1] = &w.ffn_in_t;
    for (int r = 0; r < d.nl; ++r) {
        const int deg = degree_of(r);
        const int flags = kGateSilu | (r == deg * deg ? kFirst : 0) | (r == deg * deg + 2 * deg ? kLast : 0);
        b2.tile(r * C, C, 0, deg * C, d.gates + r * C, r == 0 ? kSiluBwd : kGatedBwd, d.gates + r * C, r == 0 ? 0 : (deg - 1) * C, r == 0 ? 0 : flags);
        if (r == 0) b1.tile(0, (d.lmax + 1) * C, 0, 0, 0);
        else b1.tile((d.lmax + r) * C, C, 1, (deg - 1) * C, r * C);
    }
    const int64_t fw = (d.lmax + d.nl) * C;
    FCB_TRY(conv("ffn_out_gate_bwd", b2, L.gp.hi, L.gp.lo, row, row, b2.count(), q.ffn_y, fw, fw, &L.gy2, fw, &s->scale, &s->scale, n));
    FCB_TRY(conv("ffn_in_bwd", b1, L.gy2.hi, L.gy2.lo, fw, fw, 0, L.gxn, row, row, nullptr, 0, &s->scale, nullptr, n));
    FCB_TRY(op("rms_norm_sh_bwd", n * row * 16, [&] {
        return by_lmax([&](auto lm) {
            launch_pdl((norm_bwd_kernel<decltype(lm)::value, false>), dim3(warp_grid(n, 4)), dim3(128), 0, st, L.gxn, q.x1, w.norm2_w, q.st2, L.g, L.g1, s + 1, n);
            return 0;
        });
    }));
    // edge block
    const float* scale = &s[1].scale;
    Conv c2, c1 = blocks(w.conv1_t);
    {
        const Conv p = blocks(w.conv2_t);  // rows of one degree back to back: their gate gradient stays in registers
        c2.w[0] = p.w[0], c2.w[1] = p.w[1], c2.w[2] = p.w[2];
        auto add = [&](int r, int flags) {
            const int32_t* t = &p.t[9 * r];
            const int deg = degree_of_row(r);
            c2.tile(t[0], t[1], t[2], t[3], d.gates + r * C, r == 0 ? kSiluBwd : kGatedBwd, (r > 0 && q.a.hi ? 0 : d.gates) + r * C, r == 0 ? 0 : (deg - 1) * C, flags);
        };
        add(0, 0);
        for (int deg = 1; deg <= d.lmax; ++deg) {
            int first = 1, last = 0;
            for (int r = 1; r < d.nm; ++r)
                if (degree_of_row(r) == deg) last = r;
            for (int r = 1; r < d.nm; ++r)
                if (degree_of_row(r) == deg) {
                    add(r, (first ? kFirst : 0) | (r == last ? kLast : 0));
                    first = 0;
                }
        }
    }
    const bool first_layer = l == md.num_layers - 1;
    const Conv again = q.y ? Conv{} : conv1_gate(l, kRows);
    FCB_TRY(chunks([&](int c, int64_t e0, int64_t ec, int64_t n0, int64_t n1) {
        float* y = q.y ? q.y + e0 * q.yw : L.y_c;
        float* msg = q.msg ? q.msg + e0 * d.nm * C : L.msg_c;
        if (!q.y) {
            FCB_TRY(messages(l, again, e0, ec, y, d.yw, msg));
        } else if (!q.rad) {
            FCB_TRY(radial_out(l, e0, ec));
        }
        const float* rad = radial_of(l, e0);
        FCB_TRY(op("rotate_back_bwd", ec * 4 * (d.nl * C + 2 * d.nm * C + d.nw + 9), [&] {
            return by_lmax([&](auto lm) {
                launch_pdl((rotate_back_bwd_kernel<decltype(lm)::value, 0, OutSplit>), dim3(warp_grid(ec, 4, 148 * 12)), dim3(128), 0, st, L.g1, msg, L.wig, L.env, ev.tgt, L.gmsg.out(), scale, L.tau_e, !first_layer, 1.0f, e0, ec);
                return 0;
            });
        }));
        const Planes gated = q.a.hi ? q.a.from(e0) : Planes{};
        const int64_t yw = q.y ? q.yw : d.yw;
        FCB_TRY(conv("so2_conv_fused_conv2_gate_bwd", c2, L.gmsg.hi, L.gmsg.lo, L.gmsg.ld, L.gmsg.ld, c2.count(), y, yw, yw, &L.gy, L.gy.ld, scale, scale, ec, q.a.hi ? &gated : nullptr));
        FCB_TRY(conv("so2_conv_fused_conv1_bwd", c1, L.gy.hi, L.gy.lo, L.gy.ld, L.gy.ld, 0, L.gm, d.nm * 2 * C, d.nm * 2 * C, nullptr, 0, scale, nullptr, ec));
        const int64_t gb = ec * 4LL * (2 * d.nm * C + 2 * 2 * d.nrad * C + d.nw + 12) + (n1 - n0) * row * 4 * 4;
        FCB_TRY(op("gather_rotate_bwd", gb, [&] {
            return by_lmax([&](auto lm) {
                constexpr int LM = decltype(lm)::value;
                FCB_TRY((launch_gather_bwd<LM, 0>(*this, q.xn1, src_lo(c), src_hi(c), rad, L.gxn, c == 0, first_layer, scale, e0, 0, n)));
                return launch_gather_bwd<LM, 1>(*this, q.xn1, ev.row_ptr, ev.row_ptr + 1, rad, L.gxn, false, false, scale, e0, n0, n1);
            });
        }, 0, 2));
        return gemm("so2_conv_fused_radial_out_bwd", L.grad, w.radial_out_t, scale,
                    reinterpret_cast<float*>(L.h2) + e0 * L.rw + (int64_t)l * C, L.rw, ec);
    }));
    return op("rms_norm_sh_bwd", n * row * 16, [&] {
        return by_lmax([&](auto lm) {
            launch_pdl((norm_bwd_kernel<decltype(lm)::value, false>), dim3(warp_grid(n, 4)), dim3(128), 0, st, L.gxn, q.x0, w.norm1_w, q.st1, L.g1, L.g, s + 2, n);
            return 0;
        });
    });
}

int Run::backward() {
    const int64_t n = L.n, e = L.e;
    const int nets = L.nets, nscale = 2 * md.num_layers + 1;
    if (cudaMemsetAsync(L.scales, 0, nscale * sizeof(Scale), st) != cudaSuccess) return launch_status();
    if (!ev.grad_x) {
        FCB_TRY(op("energy_bwd", n * C * 8, [&] {
            launch_pdl(energy_bwd_kernel, dim3(warp_grid(n * C / 4, 256)), dim3(256), 0, st, L.hy2, md.head_w3, L.hg.out(), md.head_scale, n);
            return 0;
        }));
        Conv b2, b1;
        b2.w[0] = &md.head_w2_t, b1.w[0] = &md.head_w1_t;
        b2.tile(0, C, 0, 0, 0, kSiluBwd, 0);
        b1.tile(0, C, 0, 0, 0);
        // the planes of the first gradient are free once the launch that reads them is done: a row tile is written
        // after its own rows were read, but other CTAs' tiles may still be in flight, so the output goes elsewhere
        FCB_TRY(conv("head", b2, L.hg.hi, L.hg.lo, C, C, 1, L.hy1, C, C, &L.row0, C, md.head_scale, md.head_scale, n));
        FCB_TRY(conv("head", b1, L.row0.hi, L.row0.lo, C, C, 0, L.g0, C, C, nullptr, 0, md.head_scale, nullptr, n));
    }
    FCB_TRY(op("rms_norm_sh_bwd", n * d.nl * C * 8, [&] {
        return by_lmax([&](auto lm) {
            constexpr int LM = decltype(lm)::value;
            if (ev.grad_x)
                launch_pdl((norm_bwd_kernel<LM, false>), dim3(warp_grid(n, 4)), dim3(128), 0, st, ev.grad_x, L.xl, md.norm_w, L.stl, nullptr, L.g, L.scales, n);
            else
                launch_pdl((norm_bwd_kernel<LM, true>), dim3(warp_grid(n, 4)), dim3(128), 0, st, L.g0, L.xl, md.norm_w, L.stl, nullptr, L.g, L.scales, n);
            return 0;
        });
    }));
    for (int l = md.num_layers - 1; l >= 0; --l) FCB_TRY(layer_backward(l));
    // edge-degree embedding, the radial MLPs' hidden layers and the geometry, chunk by chunk
    const float* scale = &L.scales[nscale - 1].scale;
    Conv c1;
    c1.w[0] = &md.rad_w1_t;
    for (int i = 0; i < nets; ++i) c1.tile(i * C, C, 0, i * C, i * C);
    FCB_TRY(chunks([&](int, int64_t e0, int64_t ec, int64_t, int64_t) {
        FCB_TRY(degree_out(e0, ec));
        FCB_TRY(op("edge_degree_bwd", ec * 4 * (d.nl * C + 2 * (d.lmax + 1) * C + d.nw + 9), [&] {
            return by_lmax([&](auto lm) {
                launch_pdl((rotate_back_bwd_kernel<decltype(lm)::value, 1, OutSplit>), dim3(warp_grid(ec, 4, 148 * 12)), dim3(128), 0, st, L.g, L.r3, L.wig, L.env, ev.tgt, L.gr3.out(), scale, L.tau_e, 1, 1.0f / md.rescale, e0, ec);
                return 0;
            });
        }));
        float* gh = reinterpret_cast<float*>(L.h2) + e0 * L.rw;
        FCB_TRY(gemm("so2_conv_fused_radial_out_bwd", L.gr3, md.degree_out_t, scale, gh + (int64_t)md.num_layers * C, L.rw, ec));
        const int grid = warp_grid(radial_items(ec, nets, kRadialBwdRows), 8);
        FCB_TRY(op("radial_act_bwd", ec * nets * 1544, [&] {
            launch_pdl(radial_bwd_kernel, dim3(grid), dim3(256), 0, st, gh, L.pre2 + e0 * L.rw, nullptr, nullptr, ev.z, ev.src + e0, ev.tgt + e0, md.ln2_w, md.ln2_b,
                                                    L.rst2 + e0 * nets * 2, L.rp.out(), C, L.scales, nscale, L.rad_scale, ec * nets, nets);
            return 0;
        }));
        FCB_TRY(conv("so2_conv_fused_radial_in", c1, L.rp.hi, L.rp.lo, L.rw, L.rw, 0, L.rh, L.rw, L.rw, nullptr, 0, L.rad_scale, nullptr, ec));
        FCB_TRY(op("radial_act_bwd", ec * nets * 1544, [&] {
            launch_pdl(radial_bwd_kernel, dim3(grid), dim3(256), 0, st, L.rh, L.pre1 + e0 * L.rw, md.table_src, md.table_tgt, ev.z, ev.src + e0, ev.tgt + e0, md.ln1_w, md.ln1_b,
                                                    L.rst1 + e0 * nets * 2, L.rp.out(), C, L.scales, nscale, L.rad_scale, ec * nets, nets);
            return 0;
        }));
        FCB_TRY(gemm("so2_conv_fused_radial_in", L.rp, md.rad_w0_t, L.rad_scale, L.ggauss, md.num_basis, ec));
        return op("edge_geometry_bwd", ec * 4 * (md.num_basis + 9 + 4 + 8 + 3), [&] {
            return by_lmax([&](auto lm) {
                launch_pdl(geometry_bwd_kernel<decltype(lm)::value>, dim3((unsigned)((ec + 127) / 128)), dim3(128), 0, st, L.vec + e0, L.wig + e0 * d.nw, reinterpret_cast<float4*>(L.tau_n) + e0, reinterpret_cast<float4*>(L.tau_e) + e0, L.ggauss,
                    L.grad_vec + e0 * 3, basis(), ec);
                return 0;
            });
        });
    }));
    if (ev.virial) {
        const int per = e < 148 * 64 * 8 ? 8 : 128;
        FCB_TRY(op("virial", e * 28, [&] {
            launch_pdl(virial_kernel, dim3((unsigned)((e + 8 * per - 1) / (8 * per))), dim3(256), 0, st, L.grad_vec, L.vec, ev.tgt, ev.batch, ev.virial, e, per);
            return 0;
        }));
    }
    return op("grad_pos", e * 24 + n * 12, [&] {
        launch_pdl(grad_pos_kernel, dim3((unsigned)((n + 7) / 8)), dim3(256), 0, st, L.grad_vec, ev.row_ptr, ev.src_ptr, ev.src_perm, ev.grad_pos, ev.grad_sign, n);
        return 0;
    });
}

static int check(const fcb200_model* m, const fcb200_eval* e) {
    if (!m || !e || !m->layers || (m->lmax != 2 && m->lmax != 4) || m->num_layers < 1 || m->num_basis < 32 || m->num_basis % 32) return FCB200_EINVAL;
    if (m->num_layers + 1 > 40 || e->num_nodes < 1 || e->num_edges < 1 || e->num_systems < 1 || e->num_chunks < 1 || !e->chunk_node || !e->chunk_edge)
        return FCB200_EINVAL;
    if (e->chunk_edge[0] != 0 || e->chunk_edge[e->num_chunks] != e->num_edges || e->chunk_node[e->num_chunks] != e->num_nodes) return FCB200_EINVAL;
    for (int c = 0; c < e->num_chunks; ++c)
        if (e->chunk_edge[c + 1] <= e->chunk_edge[c] || e->chunk_node[c + 1] <= e->chunk_node[c]) return FCB200_EINVAL;
    return FCB200_OK;
}
static int check_call(const fcb200_model* m, const fcb200_eval* e) {
    FCB_TRY(check(m, e));
    if (!e->pos || !e->src || !e->tgt || !e->row_ptr || !e->z || !e->batch || !e->keep || !e->status) return FCB200_EINVAL;
    if (e->num_chunks > 1 && e->want_grad && !e->chunk_src) return FCB200_EINVAL;
    if ((reinterpret_cast<uintptr_t>(e->keep) | reinterpret_cast<uintptr_t>(e->scratch)) & 127) return FCB200_EALIGN;
    return FCB200_OK;
}

}  // namespace step
}  // namespace fcb200

using namespace fcb200;

extern "C" {

void fcb200_set_launch_hook(fcb200_launch_hook hook) { step::g_hook = hook; }

int fcb200_model_sizes(const fcb200_model* model, const fcb200_eval* eval, int64_t* sizes) {
    if (!sizes) return FCB200_EINVAL;
    FCB_TRY(step::check(model, eval));
    fcb200_eval e = *eval;
    e.keep = e.scratch = nullptr;
    step::Layout L;
    step::lay_out(*model, e, false, L);
    sizes[0] = L.keep_bytes, sizes[1] = L.scratch_bytes;
    step::lay_out(*model, e, true, L);
    sizes[2] = L.scratch_bytes;
    return FCB200_OK;
}

int fcb200_model_forward(const fcb200_model* model, const fcb200_eval* eval, void* stream) {
    FCB_TRY(step::check_call(model, eval));
    if (!eval->x_out || !eval->charge || !eval->spin || !eval->dataset) return FCB200_EINVAL;
    return step::Run(*model, *eval, stream, false).forward();
}

int fcb200_model_energy(const fcb200_model* model, const fcb200_eval* eval, void* stream) {
    FCB_TRY(step::check_call(model, eval));
    if (!eval->energy || !model->head_w3) return FCB200_EINVAL;
    return step::Run(*model, *eval, stream, false).energy();
}

int fcb200_model_backward(const fcb200_model* model, const fcb200_eval* eval, void* stream) {
    FCB_TRY(step::check_call(model, eval));
    if (!eval->want_grad || !eval->grad_pos || !eval->src_ptr || !eval->src_perm || (!eval->grad_x && !model->head_w3)) return FCB200_EINVAL;
    return step::Run(*model, *eval, stream, true).backward();
}

}  // extern "C"
