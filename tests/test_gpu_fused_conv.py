"""The one-launch-per-convolution kernel (gate in the epilogue) against the separate GEMM and gate kernels, which the
other GPU tests hold to the oracle: SO2_Convolution + GateActivation of the reference
(src/fairchem/core/models/uma/nn/so2_layers.py:600-647, src/fairchem/core/models/uma/nn/activation.py:146-165)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from fairchem_b200 import ops as _ops

    return _ops


def _planes(t, scale=1.0):
    t = t * scale
    hi = t.half()
    return hi, ((t - hi.float()) * 2048.0).half()


def _unplane(p, scale=1.0):
    return (p[0].float() + p[1].float() / 2048.0) / scale


@pytest.fixture(params=[0, 1, 2], ids=["per_launch_choice", "natural_groups", "row_by_row"])
def grouping(request, ops):
    """How the tile list of a launch is cut into work items.  Row by row, the gate is computed again for each row of a forward
    list; the other lists then keep their natural groups."""
    ops.CONV_GROUPING = request.param
    yield request.param
    ops.CONV_GROUPING = 0


@pytest.mark.parametrize("lmax,e", [(2, 77), (2, 1000), (4, 300), (2, 40000)])
def test_fused_convolutions_match_the_separate_kernels(ops, grouping, lmax, e):
    from fairchem_b200 import backbone as B

    torch.manual_seed(lmax)
    c = h = 128
    nm = ops.SHAPES[lmax].nm
    ew = B.Edgewise(c, h, lmax, 2, [320, 128, 128]).cuda()
    with torch.no_grad():  # biases are zero-initialised: make them count
        ew.so2_conv_1.fc_m0.bias.normal_()
        ew.so2_conv_2.fc_m0.bias.normal_()
    g = torch.Generator().manual_seed(5 + e)
    m = _planes(torch.randn(e, nm * 2 * c, generator=g).cuda())
    scale = torch.tensor([64.0], device="cuda")
    gmsg = _planes(torch.randn(e, nm * c, generator=g).cuda() * 1e-3, 64.0)
    assert B._use_fused(ew)
    with torch.no_grad():
        # separate kernels
        y_ref = B._conv_forward(ew.so2_conv_1, m)
        a_ref = B._gate(y_ref, h, nm)
        msg_ref = B._conv_forward(ew.so2_conv_2, a_ref)
        B._GemmState.a_scale = scale  # the power of two the backward operands are written with
        try:
            ga = B._conv_backward(ew.so2_conv_2, gmsg)
            gy_ref = B._new_operand(e, y_ref.shape[1], y_ref.device)
            ops.so2_gate_bwd_h_(ga, y_ref, gy_ref[0], gy_ref[1], scale, h)
            gm_ref = B._conv_backward(ew.so2_conv_1, gy_ref)
        finally:
            B._GemmState.a_scale = None
        # one launch per convolution
        y = torch.full((e, y_ref.shape[1]), float("nan"), device="cuda")
        a = B._fused_conv1_gate(ew, m, y)
        a_nokeep = B._fused_conv1_gate(ew, m, None)
        msg = B._fused_conv2(ew, a, torch.empty(e, nm * c, device="cuda"))
        gy = B._fused_conv2_gate_backward(ew, gmsg, y_ref, scale)
        gm = B._fused_conv1_backward(ew, gy, scale)
    B.check_gemm_status()
    # same arithmetic in the same order: equal up to the compiler's choice of fused multiply-adds in the gate formulas
    torch.testing.assert_close(y, y_ref, rtol=0, atol=0)
    for got, want, sc in ((a, a_ref, 1.0), (a_nokeep, a_ref, 1.0), (gy, gy_ref, 64.0)):
        ref = _unplane(want, sc)
        torch.testing.assert_close(_unplane(got, sc), ref, rtol=2e-6, atol=2e-7 * float(ref.abs().max()))
    torch.testing.assert_close(msg, msg_ref, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(gm, gm_ref, rtol=1e-5, atol=1e-5 * float(gm_ref.abs().max()))


def _launches(ops, lmax, e, form):
    """Outputs of every kind of launch, on inputs that depend on (lmax, e) alone."""
    from fairchem_b200 import backbone as B

    c, nm = 128, ops.SHAPES[lmax].nm
    torch.manual_seed(e)
    ew = B.Edgewise(c, c, lmax, 2, [320, 128, 128]).cuda()
    g = torch.Generator(device="cuda").manual_seed(7 * e + lmax)
    draw = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    m, gy = _planes(draw(e, nm * 2 * c)), _planes(draw(e, (lmax + nm) * c), 64.0)
    scale, status = torch.tensor([64.0], device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    # a list with a K tail (96 = 64 + 32), a lone tile and a last tile of 64 columns
    short, bias = draw(448, 96), draw(512)
    hi, lo, sc = ops.split_f16(short)
    tiles = [v for r in (0, 128, 256, 384) for v in (32, 96, 0, r, r, ops.CONV_PLAIN, 0, 0, 0)]
    with torch.no_grad():
        ew.so2_conv_1.fc_m0.bias.normal_()
        ew.so2_conv_2.fc_m0.bias.normal_()
        ops.CONV_GROUPING = form
        try:
            y = torch.full((e, (lmax + nm) * c), float("nan"), device="cuda")
            a = B._fused_conv1_gate(ew, m, y)
            ak = B._fused_conv1_gate(ew, m, None)
            msg = B._fused_conv2(ew, a, torch.full((e, nm * c), float("nan"), device="cuda"))
            gm = B._fused_conv1_backward(ew, gy, scale)
            gmsg = _planes(draw(e, nm * c) * 1e-3, 64.0)
            gc = B._fused_conv2_gate_backward(ew, gmsg, y, scale)
            y2 = torch.full((e, 448), float("nan"), device="cuda")
            ops.so2_conv_fused_.raw(m[0], m[1], [hi], [lo], [sc], None, tiles, 0, y2, None, None, None, None, status)
            hi, lo, sc = ops.split_f16(torch.cat([short, short[:64]]))
            y3 = torch.full((e, 512), float("nan"), device="cuda")
            ops.so2_conv_fused_.raw(m[0], m[1], [hi], [lo], [sc], bias, tiles, 0, y3, None, None, None, None, status)
        finally:
            ops.CONV_GROUPING = 0
    B.check_gemm_status()
    assert int(status) == 0
    return [y, a[0], a[1], ak[0], ak[1], msg, gm, gc[0], gc[1], y2, y3]


# one row, both sides of a warp's, a CTA's and a pair's rows; items of 32 and 64 columns (up to 1 000 rows, by the list),
# group by group (7 680) and row by row
@pytest.mark.parametrize("lmax,e", [(2, e) for e in (1, 32, 33, 128, 129, 255, 256, 257, 1000, 7680, 21000)] + [(4, 129), (4, 257), (4, 3240)])
def test_pairs_of_ctas_and_narrow_items_give_the_same_bits(ops, lmax, e):
    """Same products in the same order in every form, and every output element written."""
    alone = _launches(ops, lmax, e, 1)
    for form in (0, 3):
        for got, want in zip(_launches(ops, lmax, e, form), alone):
            assert not bool(torch.isnan(got.float()).any()) and torch.equal(got, want)


def test_pairs_of_ctas_report_values_outside_the_half_range(ops):
    """An infinite input is reported by a plain list and, through the gate, by a forward list."""
    from fairchem_b200 import backbone as B

    ew = B.Edgewise(128, 128, 2, 2, [320, 128, 128]).cuda()
    ops.CONV_GROUPING = 3
    try:
        for width, launch in ((9 * 256, lambda m: B._fused_conv1_gate(ew, m, None)),
                              (9 * 128, lambda a: B._fused_conv2(ew, a, torch.empty(300, 9 * 128, device="cuda")))):
            x = torch.randn(300, width, device="cuda")
            x[299, 5] = 1e6  # beyond 65 504: its half is infinite
            with torch.no_grad():
                launch(_planes(x))
            with pytest.raises(B.HalfRangeError):
                B.check_gemm_status()
            B.check_gemm_status()
    finally:
        ops.CONV_GROUPING = 0


def test_edge_block_is_the_same_with_and_without_the_fused_launches(ops, grouping):
    """Energy and forces of a small periodic system with the fused convolution launches on and off."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic, weights

    data = synthetic.fcc_cu((3, 3, 3), seed=1).to("cuda")
    sd = weights.random_init_state_dict(weights.UMA_S, 0)
    bb, head = B.build_model(weights.UMA_S, sd, device="cuda", edge_chunk_size=2048)
    results = []
    for fused in (True, False):
        B._GemmState.fused_conv = fused
        try:
            for keep in (0, 2):
                bb.keep_level = keep
                d = data.clone()
                out = head(d, bb(d))
                results.append((out["energy"].clone(), out["forces"].clone()))
        finally:
            B._GemmState.fused_conv = True
    e0, f0 = results[0]
    for e1, f1 in results[1:]:
        assert abs(float(e1[0] - e0[0])) <= 2e-6 * abs(float(e0[0]))
        assert float((f1 - f0).abs().max()) <= 2e-6


def test_edge_block_is_the_same_with_per_node_and_per_edge_source_gradients(ops):
    """Forces with the source half of the gather backward summed per source node inside the kernel (default) and with
    per-edge rows followed by the segmented sum (the form ``bench.py --edge-source-sums`` measures against)."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic, weights

    data = synthetic.bcc_alloy((5, 5, 5), seed=3).to("cuda")
    sd = weights.random_init_state_dict(weights.UMA_S, 0)
    bb, head = B.build_model(weights.UMA_S, sd, device="cuda", edge_chunk_size=2048)  # several chunks per layer
    results = []
    for node_sums in (True, False):
        B._GemmState.node_sums = node_sums
        try:
            d = data.clone()
            out = head(d, bb(d))
            results.append((out["energy"].clone(), out["forces"].clone()))
        finally:
            B._GemmState.node_sums = True
    (e0, f0), (e1, f1) = results
    assert abs(float(e1[0] - e0[0])) <= 1e-9 * abs(float(e0[0]))  # the forward pass is the same code
    assert float((f1 - f0).abs().max()) <= 2e-6


def _silu_list(ops, y_cols, planes, variant):
    """Status code and output planes of a list of one row-0 tile, which stores nothing to y, straight at the C entry."""
    from ctypes import c_float, c_int32, c_int64, c_void_p

    from fairchem_b200 import _lib

    m, k = 2048, 128
    g = torch.Generator(device="cuda").manual_seed(5)
    a = _planes(torch.randn(m, k, generator=g, device="cuda"))
    hi, lo, sc = ops.split_f16(torch.randn(128, k, generator=g, device="cuda"))
    y = torch.zeros(m, 128, device="cuda")
    out = [torch.zeros(m, 128, dtype=torch.float16, device="cuda") for _ in range(2)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    tiles = [0, k, 0, 0, 0, ops.CONV_SILU if planes else ops.CONV_PLAIN, 0, 0, 0]
    rc = _lib.load().fcb200_so2_conv_fused(
        a[0].data_ptr(), a[1].data_ptr(), k, k, (c_void_p * 3)(hi.data_ptr()), (c_void_p * 3)(lo.data_ptr()), (c_int64 * 3)(128), (c_int64 * 3)(k),
        (c_float * 3)(sc, 1.0, 1.0), (c_void_p * 3)(), (c_int32 * 9)(*tiles), 1, 0, y.data_ptr(), y_cols, y_cols, out[0].data_ptr(),
        out[1].data_ptr(), 128 if planes else 0, 128 if planes else 0, None, None, m, 16 * variant, status.data_ptr(),
        torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(status) == 0
    return rc, [y, *out]


@pytest.mark.parametrize("planes", [True, False])  # no column of y; planes that are passed but have no column
def test_pairs_of_ctas_take_lists_that_use_one_output(ops, planes):
    y_cols = 0 if planes else 128
    want = _silu_list(ops, y_cols, planes, 1)
    got = _silu_list(ops, y_cols, planes, 3)
    assert want[0] == got[0] == 0
    assert all(torch.equal(a, b) for a, b in zip(want[1], got[1])) and bool(got[1][1 if planes else 0].any())


# 7 680 rows: the first convolution's input alone is past the 64 MiB from which row 0 may join the group of degree 1; 21 000: the gate's
# backward too.  257: on neither.
@pytest.mark.parametrize("lmax,e", [(2, 257), (2, 7680), (2, 21000), (4, 3900), (4, 9000)])
def test_row_0_in_the_group_of_degree_1_gives_the_same_bits(ops, lmax, e):
    """Row by row (2) never joins groups, and a backward list then keeps its natural ones; the other forms may join them."""
    apart = _launches(ops, lmax, e, 2)
    for form in (0, 1, 3):
        for got, want in zip(_launches(ops, lmax, e, form), apart):
            assert torch.equal(got, want)
