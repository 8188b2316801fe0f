"""GPU parity tests of the router through the C ABI: logits bit for bit against the oracle's fixed-order fp32
definition, selections exact (ties to the lower index), routing weights within 1e-3."""
import numpy as np
import pytest

from oracle import oracle as O
from helpers import TOL_ROUTE_WEIGHT, golden, make_x, to_dev16
from router_fixtures import EXPERT_COUNTS, ROUTE_SCALE, k6_inputs, k8_inputs

pytestmark = pytest.mark.gpu


def _moe(**kw):
    from mference_b200.moe import MoE
    base = dict(d=256, f=64, num_experts=16, top_k=4, max_tokens=64)
    base.update(kw)
    return MoE(**base)


@pytest.mark.parametrize("T,E,D", [(1, 256, 2048), (2, 256, 2048), (8, 256, 2048), (64, 256, 2048), (300, 256, 2048),
                                   (5, 40, 256), (3, 33, 64), (17, 100, 4096),
                                   # above 64 rows: the lane-major fp32 kernel (d a multiple of 128; ragged row and expert
                                   # counts, fewer chunks than ring stages) and the self-contained tile kernel (d = 64)
                                   (130, 100, 1536), (1025, 256, 2048), (97, 33, 256), (70, 20, 64), (65, 1, 128)])
def test_logits_bit_exact(T, E, D):
    import torch
    W = O.LayerWeights(D, 64, E, 4, experts=[], shared=False)
    x = make_x(f"x.{T}.{E}.{D}", T, D)
    bias = np.linspace(-2, 2, E).astype(np.float32)
    moe = _moe(d=D, num_experts=E, max_tokens=T)
    xd = to_dev16(x, O.DT_BF16)
    wd = to_dev16(W.router, O.DT_BF16)
    out = torch.empty((T, E), dtype=torch.float32, device="cuda")
    for lb in (None, bias):
        moe.encode_router_logits(xd, wd, out, None if lb is None else torch.from_numpy(lb).cuda())
        ref = O.router_logits(x, O.DT_BF16, W.router, logit_bias=lb)
        got = out.cpu().numpy()
        assert (got.view(np.uint32) == ref.view(np.uint32)).all(), np.abs(got - ref).max()


def test_logits_fp16_activations_and_row_stride():
    import torch
    T, E, D = 6, 24, 128
    W = O.LayerWeights(D, 64, E, 4, experts=[], shared=False)
    x = make_x("x16", T, D, dtype=O.DT_F16)
    from mference_b200 import DT_F16
    moe = _moe(d=D, num_experts=E, max_tokens=T, x_dtype=DT_F16)
    wide = torch.zeros((T, D + 64), dtype=torch.float16, device="cuda")
    wide[:, :D] = to_dev16(x, O.DT_F16)
    out = torch.empty((T, E), dtype=torch.float32, device="cuda")
    moe.encode_router_logits(wide[:, :D], to_dev16(W.router, O.DT_BF16), out)
    ref = O.router_logits(x, O.DT_F16, W.router)
    assert (out.cpu().numpy().view(np.uint32) == ref.view(np.uint32)).all()


def test_logits_many_rows_fp16_activations_and_row_stride():
    import torch
    T, E, D = 97, 48, 512
    W = O.LayerWeights(D, 64, E, 4, experts=[], shared=False)
    x = make_x("x16.many", T, D, dtype=O.DT_F16)
    from mference_b200 import DT_F16
    moe = _moe(d=D, num_experts=E, max_tokens=T, x_dtype=DT_F16)
    wide = torch.zeros((T, D + 72), dtype=torch.float16, device="cuda")
    wide[:, :D] = to_dev16(x, O.DT_F16)
    out = torch.empty((T, E), dtype=torch.float32, device="cuda")
    moe.encode_router_logits(wide[:, :D], to_dev16(W.router, O.DT_BF16), out)
    ref = O.router_logits(x, O.DT_F16, W.router)
    assert (out.cpu().numpy().view(np.uint32) == ref.view(np.uint32)).all()


@pytest.mark.parametrize("T,E,D,K", [(203, 256, 2048, 8), (593, 256, 2048, 8), (640, 256, 4096, 6), (2400, 33, 256, 4), (330, 500, 512, 16),
                                     (4800, 7, 2304, 8), (1190, 256, 512, 8), (1251, 300, 4096, 6)])
@pytest.mark.parametrize("x_dtype", ["bf16", "f16"])
@pytest.mark.parametrize("mode", ["softmax", "sqrtsoftplus"])
def test_topk_of_a_block_equals_ordered_logits_and_select_bit_for_bit(T, E, D, K, x_dtype, mode):
    """Large blocks of rows form the ordered logits only for the experts that can win.  Same indices and weights as all
    ordered logits followed by the selection - with exact ties (equal gate rows, zero token rows), near ties, a gate row
    far larger than the others, values beyond the fp16 range and infinities, rows so small that their squares vanish in fp32, and
    gate rows that differ in one small element only, all of one sign and parallel to a token row (the sum of the magnitudes is
    then as large as the norms allow)."""
    import torch
    from mference_b200 import DT_BF16, DT_F16, ROUTER_SOFTMAX_TOPK, ROUTER_SQRTSOFTPLUS
    from mference_b200.moe import MoELayerWeights
    from mference_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(T + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    moe = _moe(d=D, num_experts=E, top_k=K, max_tokens=T, x_dtype=DT_BF16 if x_dtype == "bf16" else DT_F16,
               router_mode=ROUTER_SOFTMAX_TOPK if mode == "softmax" else ROUTER_SQRTSOFTPLUS, route_scale=1.5)
    x = rnd(T, D).to(torch.bfloat16 if x_dtype == "bf16" else torch.float16)
    x[3] = 0
    x[5] = x[6]
    if x_dtype == "bf16":
        x[7:20] = (x[7:20].float() * 2.0 ** -85).to(torch.bfloat16)
        x[20:30] = (x[20:30].float() * 2.0 ** -60).to(torch.bfloat16)
    gate = (rnd(E, D) * 0.05).to(torch.bfloat16)
    gate[2] = gate[4]
    gate[5] = gate[4] * (1 + 2.0 ** -7)
    variants = {"plain": gate, "large": gate.clone(), "beyond": gate.clone(), "inf": gate.clone()}
    variants["large"][1] *= 1000
    variants["beyond"][3, 0] = 3.0e5
    variants["inf"][0, 7] = float("inf")
    twins = gate[:1].abs().repeat(E, 1)
    twins[:, :E] = 0
    twins[torch.arange(E), torch.arange(E)] = (torch.arange(E, device="cuda") % 64 * 2.0 ** -23).to(torch.bfloat16)
    variants["twins"] = twins
    if x_dtype == "bf16":
        variants["tiny"] = (gate.float() * 2.0 ** -70).to(torch.bfloat16)
        variants["tiny twins"] = (twins.float() * 2.0 ** -70).to(torch.bfloat16)
    x[30:40] = (20 * gate[:1].abs().float() * (1 + 0.1 * rnd(10, D).abs())).to(x.dtype)
    bias = rnd(E).float()
    scale = (1 + 0.1 * rnd(E)).to(torch.bfloat16)
    corr = rnd(E).float() * 0.1
    logits = torch.empty((T, E), dtype=torch.float32, device="cuda")
    got_i, want_i = (torch.zeros((T, K), dtype=torch.int32, device="cuda") for _ in range(2))
    got_w, want_w = (torch.zeros((T, K), dtype=torch.float16, device="cuda") for _ in range(2))
    for name, w in variants.items():
        for lb in (None, bias):
            lw = MoELayerWeights(router_w=w, pool=w, slot_stride=0, routed_off=L.ExpertOffsets(), logit_bias=lb,
                                 per_expert_scale=scale if mode == "softmax" else None,
                                 correction_bias=corr if mode == "sqrtsoftplus" else None)
            moe.encode_router(x, lw, got_i, got_w)
            moe.encode_router_logits(x, w, logits, lb)
            moe.encode_router_select(logits, want_i, want_w, per_expert_scale=lw.per_expert_scale, correction_bias=lw.correction_bias)
            assert torch.equal(got_i, want_i), name
            assert torch.equal(got_w.view(torch.int16), want_w.view(torch.int16)), name
    assert moe.device_status() == 0


def test_block_of_rows_equals_single_rows_bit_for_bit():
    # PrefillRouterTests: the block router equals the repeated single-row router
    import torch
    T, E, D, K = 19, 256, 2048, 8
    W = O.LayerWeights(D, 64, E, K, experts=[], shared=False)
    x = to_dev16(make_x("xb", T, D), O.DT_BF16)
    wd = to_dev16(W.router, O.DT_BF16)
    moe = _moe(d=D, num_experts=E, top_k=K, max_tokens=T)
    block = torch.empty((T, E), dtype=torch.float32, device="cuda")
    moe.encode_router_logits(x, wd, block)
    single = torch.empty((T, E), dtype=torch.float32, device="cuda")
    for t in range(T):
        moe.encode_router_logits(x[t:t + 1], wd, single[t:t + 1])
    assert torch.equal(block.view(torch.int32), single.view(torch.int32))


def test_calls_that_begin_with_the_gate_see_what_the_kernel_in_front_wrote():
    """The gate kernels request the gate before the kernel in front has ended; as a call's first kernel they must not, since that
    kernel may be the caller's and write the gate: here a copy kernel does, for each of the four entry points in turn."""
    import ctypes as C
    import torch
    from mference_b200 import _lib as L
    from mference_b200.moe import MoELayerWeights, encode_router_static, expert_layout
    E, D, K, T = 256, 2048, 8, 4
    gen = torch.Generator(device="cuda").manual_seed(9)
    gates = [torch.randn((E, D), device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2)]
    codes = [torch.randint(0, 256, (E, D), device="cuda", generator=gen, dtype=torch.uint8) for _ in range(2)]
    sb = torch.full((E, D // 64), 0.01, device="cuda").to(torch.bfloat16)
    x = torch.randn((T, D), device="cuda", generator=gen).to(torch.bfloat16)
    moe = _moe(d=D, f=512, num_experts=E, top_k=K, max_tokens=T)
    gate, code = torch.empty_like(gates[0]), torch.empty_like(codes[0])
    lw = MoELayerWeights(router_w=gate, pool=torch.zeros(16, dtype=torch.uint8, device="cuda"), slot_stride=16, routed_off=expert_layout(4, D, 512)[0])
    logits, y = (torch.empty((T, E), device="cuda") for _ in range(2))
    out = [(torch.empty((T, K), dtype=torch.int32, device="cuda"), torch.empty((T, K), dtype=torch.float16, device="cuda")) for _ in range(2)]
    stream = lambda: C.c_void_p(torch.cuda.current_stream().cuda_stream)
    calls = [lambda: moe.encode_router_logits(x, gate, logits), lambda: moe.encode_router(x, lw, *out[0]),
             lambda: encode_router_static(x, gate, *out[1], top_k=K),
             lambda: L.check(L.load().mfb_gemv_int8(stream(), code.data_ptr(), sb.data_ptr(), sb.data_ptr(), x.data_ptr(), L.DT_BF16, D, T, None, E, D, y.data_ptr()))]

    def run(i, wait):
        for call in calls:
            for dst, src in ((gate, gates), (code, codes)):
                dst.zero_()
                torch.add(src[i], 0, out=dst)
            if wait:
                torch.cuda.synchronize()
            call()
        torch.cuda.synchronize()
        return [t.clone() for t in (logits, y, *out[0], *out[1])]

    want = [run(i, True) for i in range(2)]
    for n in range(20):
        assert all(torch.equal(a, b) for a, b in zip(run(n % 2, False), want[n % 2])), n


def test_static_router_without_a_handle_on_the_device():
    """mfb_router_topk_static needs no handle; without one on its device the kernels have not been given more than 48 KB of shared
    memory there and take fewer rows at a time.  A fresh process routes first, then creates a handle: the same bits."""
    import subprocess
    import sys
    code = """if 1:
        import torch
        from mference_b200.moe import MoE, MoELayerWeights, encode_router_static, expert_layout
        for T, D in ((1, 4096), (8, 4096), (64, 4096), (8, 2048), (3, 8192), (64, 2048)):
            gen = torch.Generator(device="cuda").manual_seed(T)
            x = torch.randn((T, D), device="cuda", generator=gen).to(torch.bfloat16)
            gate = torch.randn((40, D), device="cuda", generator=gen).to(torch.bfloat16)
            new = lambda: (torch.zeros((T, 6), dtype=torch.int32, device="cuda"), torch.zeros((T, 6), dtype=torch.float16, device="cuda"))
            globals().setdefault("first", {})[T, D] = (x, gate, new())
            encode_router_static(x, gate, *first[T, D][2], top_k=6)
        for (T, D), (x, gate, got) in first.items():
            moe = MoE(D, 64, 40, 6, max_tokens=T)
            lw = MoELayerWeights(router_w=gate, pool=torch.zeros(16, dtype=torch.uint8, device="cuda"), slot_stride=16, routed_off=expert_layout(4, D, 64)[0])
            want = [t.clone() for t in got], [torch.empty_like(t) for t in got]
            moe.encode_router(x, lw, *want[1])
            encode_router_static(x, gate, *got, top_k=6)
            assert all(torch.equal(a, b) and torch.equal(a, c) for a, b, c in zip(got, *want)), (T, D)
            moe.close()
        print("same")
    """
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=240)
    assert done.stdout.strip() == "same", done.stderr[-2000:]


def test_select_golden_tie_fixtures():
    import torch
    from mference_b200 import ROUTER_SQRTSOFTPLUS
    cases = {(c["mode"], c["num_experts"], c["trial"]): c for c in golden("router_topk_cases.json")["cases"]}
    for ne in EXPERT_COUNTS:
        moe8 = _moe(num_experts=ne, top_k=8, max_tokens=16)
        lgs, scales = zip(*[(lg, sc) for _, lg, sc in k8_inputs(ne)])
        idx = torch.empty((len(lgs), 8), dtype=torch.int32, device="cuda")
        w = torch.empty((len(lgs), 8), dtype=torch.float16, device="cuda")
        for trial, (lg, sc) in enumerate(zip(lgs, scales)):
            moe8.encode_router_select(torch.from_numpy(lg[None]).cuda(), idx[trial:trial + 1], w[trial:trial + 1],
                                      per_expert_scale=to_dev16(O.f32_to_bf16(sc), O.DT_BF16))
        for trial in range(len(lgs)):
            c = cases[("softmax_k8", ne, trial)]
            assert idx[trial].tolist() == c["indices"], (ne, trial)
            assert np.abs(w[trial].float().cpu().numpy() - np.array(c["weights"])).max() < TOL_ROUTE_WEIGHT
            oi, ow = O.topk_softmax(lgs[trial][None], 8, O.f32_to_bf16(scales[trial]))
            assert idx[trial].tolist() == oi[0].tolist()
        moe6 = _moe(num_experts=ne, top_k=6, max_tokens=16, router_mode=ROUTER_SQRTSOFTPLUS, route_scale=ROUTE_SCALE)
        for trial, lg, bias in k6_inputs(ne):
            i6 = torch.empty((1, 6), dtype=torch.int32, device="cuda")
            w6 = torch.empty((1, 6), dtype=torch.float16, device="cuda")
            moe6.encode_router_select(torch.from_numpy(lg[None]).cuda(), i6, w6, correction_bias=torch.from_numpy(bias).cuda())
            c = cases[("sqrtsoftplus_k6", ne, trial)]
            assert i6[0].tolist() == c["indices"], (ne, trial)
            assert np.abs(w6[0].float().cpu().numpy() - np.array(c["weights"])).max() < 2e-3


def test_select_fewer_experts_than_k():
    import torch
    moe = _moe(num_experts=3, top_k=8, max_tokens=1)
    lg = torch.tensor([[0.5, 1.5, 1.0]], dtype=torch.float32, device="cuda")
    idx = torch.empty((1, 8), dtype=torch.int32, device="cuda")
    w = torch.empty((1, 8), dtype=torch.float16, device="cuda")
    moe.encode_router_select(lg, idx, w)
    assert idx[0].tolist() == [1, 2, 0, 0, 0, 0, 0, 0]
    assert float(w[0, 3:].float().abs().max()) == 0.0


@pytest.mark.parametrize("T", [1, 8, 64, 4096])
def test_router_topk_exact_at_qwen_shape(T):
    import torch
    E, D, K = 256, 2048, 8
    W = O.LayerWeights(D, 64, E, K, experts=[], shared=False)
    x = make_x(f"xq{T}", T, D)
    from mference_b200.moe import MoELayerWeights, expert_layout
    moe = _moe(d=D, f=512, num_experts=E, top_k=K, max_tokens=T)
    off, _ = expert_layout(4, D, 512)
    lw = MoELayerWeights(router_w=to_dev16(W.router, O.DT_BF16), pool=torch.zeros(16, dtype=torch.uint8, device="cuda"),
                         slot_stride=16, routed_off=off)
    idx = torch.empty((T, K), dtype=torch.int32, device="cuda")
    w = torch.empty((T, K), dtype=torch.float16, device="cuda")
    moe.encode_router(to_dev16(x, O.DT_BF16), lw, idx, w)
    lg = O.router_logits(x, O.DT_BF16, W.router)
    oi, ow = O.topk_softmax(lg, K)
    assert (idx.cpu().numpy().astype(np.uint32) == oi).all()
    assert np.abs(w.float().cpu().numpy() - O.f16_to_f32(ow)).max() < TOL_ROUTE_WEIGHT
    # the fixed summation order does not hide a wrong answer: wherever the exact (double) logits separate the
    # candidates by more than fp32 noise, the selection is the same
    lg64 = O.router_logits(x, O.DT_BF16, W.router, exact_f64=True)
    clear = O.topk_margin(lg64, K) > 1e-4
    oi64, _ = O.topk_softmax(lg64, K)
    assert (idx.cpu().numpy().astype(np.uint32)[clear] == oi64[clear]).all()
    assert clear.mean() > 0.95


def test_slot_lookup():
    import torch
    moe = _moe(num_experts=16, top_k=4, max_tokens=8)
    table = torch.full((16,), -1, dtype=torch.int16, device="cuda")
    table[3], table[5], table[7], table[9] = 0, 2, 1, 3
    idx = torch.tensor([[3, 5, 7, 9], [3, 4, 7, 9], [99, 3, 5, 7]], dtype=torch.int32, device="cuda")
    offs = torch.empty((3, 4), dtype=torch.int64, device="cuda")
    hit = torch.empty(3, dtype=torch.int32, device="cuda")
    moe.encode_slot_lookup(idx, table, 1000, offs, hit)
    assert hit.tolist() == [1, 0, 0]        # row 2: index clamped to the last expert, which is not resident
    assert offs[0].tolist() == [0, 2000, 1000, 3000] and offs[1].tolist() == [0, 0, 1000, 3000]


@pytest.mark.parametrize("T,E,D", [(65, 256, 256), (144, 250, 512), (145, 256, 128), (288, 250, 256), (289, 33, 128), (600, 40, 128)])
def test_logits_of_a_block_in_tiles_of_eight_sixteen_and_32_rows(T, E, D):
    """The tile halves while SMs would be idle: the same bits on either side of both limits (18 tiles of rows by 8 of experts), with
    rows and experts that do not fill a tile."""
    import torch
    x = make_x("x.tiles", T, D)
    w = make_x("w.tiles", E, D, std=0.02)
    moe = _moe(d=D, num_experts=E, max_tokens=T)
    xd, wd = to_dev16(x, O.DT_BF16), to_dev16(w, O.DT_BF16)
    out = torch.empty((T, E), dtype=torch.float32, device="cuda")
    moe.encode_router_logits(xd, wd, out)
    ref = O.router_logits(x, O.DT_BF16, w)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("T,E,D", [(2, 33, 64), (3, 33, 2048), (4, 250, 256), (5, 255, 2048), (7, 33, 8192), (9, 250, 4096), (16, 33, 256), (17, 255, 2048),
                                   (23, 250, 4096), (64, 33, 2048), (25, 33, 4224)])
def test_logits_of_a_few_rows_spread_over_warps(T, E, D):
    """Rows and experts that do not fill a block's warps, and gate rows of which two, four or eight token rows fit shared memory: the same bits."""
    import torch
    x = make_x("x.warps", T, D)
    w = make_x("w.warps", E, D, std=0.02)
    moe = _moe(d=D, num_experts=E, max_tokens=T)
    xd, wd = to_dev16(x, O.DT_BF16), to_dev16(w, O.DT_BF16)
    out = torch.empty((T, E), dtype=torch.float32, device="cuda")
    moe.encode_router_logits(xd, wd, out)
    ref = O.router_logits(x, O.DT_BF16, w)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32))
