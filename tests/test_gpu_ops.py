"""GPU parity of the operator table against the CPU oracle and the golden fixtures.
Every call goes through the C-ABI library (ctypes); tolerances are the reference's own
(rtol 0.02 / atol 0.002 on bf16 outputs, 2e-5 / 1e-6 on the fp32 state) plus the 1e-2
relative-L2 bound against an fp32-dequantised product."""

import pytest
import torch

from oracle import decode_oracle as O
from quickdraw_b200 import synthetic
from quickdraw_b200.synthetic import to_device
from quickdraw_b200.weights import NVFP4Linear
from tests.golden.fixture_io import from_tree

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K(cuda_device):
    from quickdraw_b200 import kernels
    return kernels


def close(actual, expected, rtol=0.02, atol=0.002):
    torch.testing.assert_close(actual.float().cpu(), expected.float().cpu(), rtol=rtol, atol=atol)


# ----------------------------------------------------------------------------- formats
def test_dequant_all_codes_all_scales_bit_exact(K, cuda_device):
    scale_codes = [c for c in range(256) if (c & 0x7F) != 0x7F]
    rows = len(scale_codes)
    codes = torch.arange(256, dtype=torch.int32).to(torch.uint8).repeat(rows, 1)          # in = 512
    scales = torch.tensor(scale_codes, dtype=torch.uint8).view(torch.float8_e4m3fn).reshape(rows, 1).repeat(1, 32)
    proj = NVFP4Linear(codes, scales.contiguous(), torch.tensor(1.0))
    expected = O.dequantize_fp32(proj)
    dev = to_device(proj, cuda_device)
    for hardware in (False, True):
        got = K.dequantize(dev, hardware_convert=hardware).cpu()
        assert torch.equal(got, expected)
        assert torch.equal(torch.signbit(got), torch.signbit(expected))


# ------------------------------------------------------------------------------ matvec
def test_gemv_golden_cases(K, cuda_device, reference_outputs):
    for case in from_tree(reference_outputs["gemv"]):
        x, proj = case["x"].to(cuda_device), to_device(case["proj"], cuda_device)
        routing = case["routing"]
        for generic in (True, False):
            got = K.nvfp4_gemv(x, proj, routing_weight=None if routing is None else routing.to(cuda_device),
                               force_generic=generic)
            close(got, case["expected"])
    case = from_tree(reference_outputs["all_codes"])
    close(K.nvfp4_gemv(case["x"].to(cuda_device), to_device(case["proj"], cuda_device)), case["expected"])


def test_routed_double_rounding_known_answer(K, cuda_device, reference_outputs):
    case = from_tree(reference_outputs["routed_kat"])
    got = K.nvfp4_gemv(case["x"].to(cuda_device), to_device(case["proj"], cuda_device),
                       routing_weight=case["routing"].to(cuda_device))
    assert got.item() == 5.5625


@pytest.mark.parametrize("rows,width", [(1024, 2048), (2048, 4096), (333, 2048), (8192, 2048), (77, 4096)])
def test_streaming_gemv_matches_oracle(K, cuda_device, rows, width):
    torch.manual_seed(rows + width)
    x = torch.randn(width).bfloat16()
    codes = torch.randint(0, 256, (rows, width // 2), dtype=torch.uint8)
    scales = (torch.randn(rows, width // 16).abs() * 0.05).to(torch.float8_e4m3fn)
    proj = NVFP4Linear(codes, scales, torch.tensor(0.75))
    expected = O.nvfp4_gemv(x, proj)
    got = K.nvfp4_gemv(x.to(cuda_device), to_device(proj, cuda_device))
    close(got, expected)
    assert O.rel_l2(got.cpu(), O.fp32_dequant_matvec(x, proj)) < 1e-2
    generic = K.nvfp4_gemv(x.to(cuda_device), to_device(proj, cuda_device), force_generic=True)
    close(generic, expected)
    # the two CUDA paths differ only in fp32 summation order
    assert O.rel_l2(got.cpu(), generic.cpu()) < 4e-3


def test_config1_single_matvec(K, cuda_device, reference_outputs):
    case = from_tree(reference_outputs["config1_head"])
    x, proj = synthetic.matvec_case(0)
    got = K.nvfp4_gemv(x.to(cuda_device), to_device(proj, cuda_device)).cpu()
    close(got[:case["rows"]], case["expected"])
    close(got, O.nvfp4_gemv(x, proj))
    assert O.rel_l2(got, O.fp32_dequant_matvec(x, proj)) < 1e-2


def test_large_activations_do_not_overflow_f16(K, cuda_device):
    torch.manual_seed(3)
    x = (torch.randn(2048) * 3.0e5).bfloat16()
    proj = synthetic.Source(1, "cpu").nvfp4("big", 64, 2048)
    got = K.nvfp4_gemv(x.to(cuda_device), to_device(proj, cuda_device))
    want = O.nvfp4_gemv(x, proj)
    assert torch.isfinite(got).all()
    assert O.rel_l2(got.cpu(), want) < 1e-2


def test_expert_bank_cases(K, cuda_device, reference_outputs):
    for case in from_tree(reference_outputs["expert_gemv"]):
        got = K.expert_gemv(case["x"].to(cuda_device), to_device(case["proj"], cuda_device),
                            case["ids"].to(cuda_device),
                            None if case["routing"] is None else case["routing"].to(cuda_device))
        close(got, case["expected"])


def test_gate_up_plain_and_bank(K, cuda_device):
    src = synthetic.Source(9, "cpu")
    x = src.normal("x", 2048)
    for experts in (None, 6):
        gate, up = src.nvfp4("g", 96, 2048, experts), src.nvfp4("u", 96, 2048, experts)
        ids = None if experts is None else torch.tensor([5, 0, 3], dtype=torch.int32)
        if experts is None:
            want = O.swiglu(O.nvfp4_gemv(x, gate), O.nvfp4_gemv(x, up))
        else:
            want = torch.stack([O.swiglu(O.nvfp4_gemv(x, O.expert_view(gate, e)), O.nvfp4_gemv(x, O.expert_view(up, e)))
                                for e in ids.tolist()])
        for generic in (False, True):
            got = K.gate_up(x.to(cuda_device), to_device(gate, cuda_device), to_device(up, cuda_device),
                            None if ids is None else ids.to(cuda_device), force_generic=generic)
            close(got, want)


def test_bf16_gemv_and_fp8_gemv(K, cuda_device):
    torch.manual_seed(5)
    x = torch.randn(2048).bfloat16()
    w = (torch.randn(300, 2048) * 0.02).bfloat16()
    close(K.bf16_gemv(x.to(cuda_device), w.to(cuda_device)), O.bf16_gemv(x, w))
    from quickdraw_b200.weights import FP8Linear
    eye = FP8Linear(torch.eye(3).to(torch.float8_e4m3fn), torch.tensor(1.0), torch.tensor(1.0))
    got = K.fp8_gemv(torch.tensor([1.0625, 1.1875, -1.0625], device=cuda_device), to_device(eye, cuda_device))
    assert got.cpu().tolist() == [1.0, 1.25, -1.0]       # ties round to even
    proj = FP8Linear((torch.randn(40, 96) * 0.5).to(torch.float8_e4m3fn), torch.tensor(0.125), torch.tensor(0.25))
    xs = torch.randn(96).bfloat16()
    close(K.fp8_gemv(xs.to(cuda_device), to_device(proj, cuda_device)), O.fp8_gemv(xs, proj))


def test_rms_norm(K, cuda_device):
    torch.manual_seed(6)
    for dtype in (torch.bfloat16, torch.float32):
        x = torch.randn(5, 2048).to(dtype)
        gamma = 1 + torch.randn(2048) * 0.1
        got = K.rms_norm(x.to(cuda_device), gamma.to(cuda_device), 1e-6)
        close(got, O.rms_norm(x, gamma, 1e-6), rtol=0.016 if dtype == torch.bfloat16 else 2e-5, atol=1e-6)
    x, r = torch.randn(2048).bfloat16(), torch.randn(2048).bfloat16()
    normed, res = K.add_rms_norm(x.to(cuda_device), r.to(cuda_device), gamma.to(cuda_device), 1e-6)
    want_n, want_r = O.add_norm(x, r, gamma, 1e-6)
    close(normed, want_n, rtol=0.016, atol=1e-6)
    assert torch.equal(res.cpu(), want_r)


# ----------------------------------------------------------------------------- routing
def test_route_ids_exact(K, cuda_device, reference_outputs):
    for case in from_tree(reference_outputs["route"]):
        ids, weights = K.route(case["logits"].to(cuda_device), case["topk"])
        assert torch.equal(ids.cpu(), case["ids"])
        torch.testing.assert_close(weights.cpu(), case["weights"], rtol=2e-6, atol=1e-7)


# --------------------------------------------------------------------------------- MoE
def test_moe_golden(K, cuda_device, reference_outputs):
    ckpt = from_tree(reference_outputs["mini_ckpt"])
    case = from_tree(reference_outputs["moe"])
    got = K.moe_block(to_device(ckpt.layers[0].moe, cuda_device), case["x"].to(cuda_device), config=ckpt.config)
    close(got, case["expected"])
    ties = from_tree(reference_outputs["moe_ties"])
    close(K.moe_block(to_device(ties["w"], cuda_device), ties["x"].to(cuda_device), config=ckpt.config), ties["expected"])


def test_moe_layer_full_width(K, cuda_device):
    """One MoE layer of the 36B-A3B shape (256 experts, top-8, intermediate 512)."""
    cfg = synthetic.model_config(num_layers=1)
    src = synthetic.Source(2, cuda_device)
    moe = synthetic.make_moe(cfg, src)
    x = src.normal("x", cfg.hidden_size)
    got = K.moe_block(moe, x, config=cfg).cpu()
    want = O.moe_block(to_device(moe, "cpu"), x.cpu(), config=cfg)
    close(got, want)
    assert O.rel_l2(got, want) < 1e-2
    logits = K.bf16_gemv(x, moe.router)
    ids, _ = K.route(logits, cfg.num_experts_per_tok)
    want_ids, _ = O.route(O.bf16_gemv(x.cpu(), moe.router.cpu()), cfg.num_experts_per_tok)
    assert torch.equal(ids.cpu(), want_ids)


# ------------------------------------------------------------------------------ mixers
def test_gdn_golden(K, cuda_device, reference_outputs):
    ckpt = from_tree(reference_outputs["mini_ckpt"])
    data = from_tree(reference_outputs["gdn"])
    w = to_device(ckpt.layers[0].attn, cuda_device)
    rec, conv = data["rec0"].to(cuda_device), data["conv0"].to(cuda_device)
    for step, entry in enumerate(data["steps"]):
        got = K.gated_delta_net_block(w, entry["x"].to(cuda_device), rec, conv, step, config=ckpt.config)
        close(got, entry["expected"])
        assert torch.equal(conv.cpu(), entry["conv_after"])
    torch.testing.assert_close(rec.cpu(), data["rec_after"], rtol=1e-3, atol=1e-5)


def test_gdn_full_width(K, cuda_device):
    cfg = synthetic.model_config(num_layers=1)
    src = synthetic.Source(4, cuda_device)
    w = synthetic.make_gdn(cfg, src)
    rec = (torch.randn(32, 128, 128, device=cuda_device) * 0.01)
    conv = src.normal("conv", cfg.conv_channels, 3)
    rec_c, conv_c, w_c = rec.cpu().clone(), conv.cpu().clone(), to_device(w, "cpu")
    for step in range(2):
        x = src.normal(f"x{step}", cfg.hidden_size)
        got = K.gated_delta_net_block(w, x, rec, conv, step, config=cfg)
        want = O.gated_delta_net_block(w_c, x.cpu(), rec_c, conv_c, step, config=cfg)
        assert O.rel_l2(got.cpu(), want) < 1e-2
        close(got, want, rtol=0.05, atol=0.05)
    assert O.rel_l2(rec.cpu(), rec_c) < 1e-3
    assert O.rel_l2(conv.cpu(), conv_c) < 1e-2


def test_attention_golden(K, cuda_device, reference_outputs):
    ckpt = from_tree(reference_outputs["mini_ckpt"])
    data = from_tree(reference_outputs["attention"])
    w = to_device(ckpt.layers[1].attn, cuda_device)
    for case in data["cases"]:
        k, v = data["k"].to(cuda_device), data["v"].to(cuda_device)
        got = K.full_attention_block(w, case["x"].to(cuda_device), (k, v), case["position"], config=ckpt.config)
        close(got, case["expected"])
        p = case["position"]
        close(k[p], case["k_row"])
        assert torch.equal(v[p].cpu(), case["v_row"])
        others = [i for i in range(k.shape[0]) if i != p]
        assert torch.equal(k[others].cpu(), data["k"][others]) and torch.equal(v[others].cpu(), data["v"][others])
        # device-scalar position gives the same result
        k2, v2 = data["k"].to(cuda_device), data["v"].to(cuda_device)
        pos = torch.tensor(p, dtype=torch.int32, device=cuda_device)
        again = K.full_attention_block(w, case["x"].to(cuda_device), (k2, v2), pos, config=ckpt.config)
        assert torch.equal(again, got)


@pytest.mark.parametrize("position", [0, 63, 64, 700, 4095])
def test_attention_full_width(K, cuda_device, position):
    cfg = synthetic.model_config(num_layers=4)
    src = synthetic.Source(8, cuda_device)
    w = synthetic.make_attention(cfg, src)
    capacity = 4096
    k = src.normal("k", capacity, 2, 256)
    v = src.normal("v", capacity, 2, 256)
    x = src.normal("x", cfg.hidden_size)
    kc, vc = k.cpu().clone(), v.cpu().clone()
    got = K.full_attention_block(w, x, (k, v), position, config=cfg)
    want = O.full_attention_block(to_device(w, "cpu"), x.cpu(), (kc, vc), position, config=cfg)
    assert O.rel_l2(got.cpu(), want) < 1e-2
    assert O.rel_l2(k[position].cpu(), kc[position]) < 1e-2
    assert torch.equal(v[position].cpu(), vc[position])


@pytest.mark.parametrize("capacity,position", [(8192, 8191), (8192, 5000), (32768, 32767), (32768, 20011)])
def test_attention_long_context(K, cuda_device, capacity, position):
    """The attention configurations of the baseline: 16 query / 2 KV heads of 256, bf16 cache of
    8192 and 32768 positions ~ N(0, 1), decode at the last position and at one in the middle;
    against the oracle within 1e-2 relative L2 (fp32 softmax over the whole history on the CPU)."""
    cfg = synthetic.model_config(num_layers=4)
    src = synthetic.Source(9, cuda_device)
    w = synthetic.make_attention(cfg, src)
    k = src.normal("k", capacity, 2, 256)
    v = src.normal("v", capacity, 2, 256)
    x = src.normal("x", cfg.hidden_size)
    kc, vc = k.cpu().clone(), v.cpu().clone()
    got = K.full_attention_block(w, x, (k, v), position, config=cfg)
    want = O.full_attention_block(to_device(w, "cpu"), x.cpu(), (kc, vc), position, config=cfg)
    assert O.rel_l2(got.cpu(), want) < 1e-2
    assert O.rel_l2(k[position].cpu(), kc[position]) < 1e-2
    assert torch.equal(v[position].cpu(), vc[position])
    untouched = [position - 1, 0] if position else []
    for t in untouched:
        assert torch.equal(k[t].cpu(), kc[t]) and torch.equal(v[t].cpu(), vc[t])


@pytest.mark.parametrize("hq,hk,rotary", [(16, 2, 64), (3, 1, 128), (8, 8, 0), (10, 2, 256)])
@pytest.mark.parametrize("position", [0, 1, 15, 16, 127, 128, 255, 256, 511, 4097])
def test_attention_tensor_core_form_at_the_edges_of_its_chunks(cuda_device, hq, hk, rotary, position):
    """Head dimension 256 with every group size class and rotary width: contexts that end on either side of a chunk of
    sixteen, of a round of eight warps and of a split, few splits and many, rows past the position poisoned, position from
    the host and from the device.  Bound: the operands are bf16 and exact in the oracle, sums fp32, one rounding of the
    result and one of the gated product: 2 ulp of bf16."""
    from quickdraw_b200._lib import call, lib, ptr, stream_of
    d, cap, eps, theta = 256, 4200, 1e-6, 1.0e7
    src = synthetic.Source(77, "cpu")
    qg, k_new, v_new = src.normal("qg", hq, 2 * d), src.normal("k", hk, d), src.normal("v", hk, d)
    q_norm, k_norm = src.normal("qn", d, std=0.1), src.normal("kn", d, std=0.1)
    kc, vc = src.normal("kc", cap, hk, d), src.normal("vc", cap, hk, d)
    kc[position:], vc[position:] = float("nan"), float("nan")
    cos, sin = O.rope_tables(position, rotary, theta)
    q = O.apply_rope(O.rms_norm(qg[:, :d], 1 + q_norm.float(), eps), cos, sin)
    wk, wv = kc.clone(), vc.clone()
    wk[position], wv[position] = O.apply_rope(O.rms_norm(k_new, 1 + k_norm.float(), eps), cos, sin), v_new
    keys, values = (t[:position + 1].double().repeat_interleave(hq // hk, 1) for t in (wk, wv))
    p = torch.softmax(torch.einsum("hd,thd->ht", q.double(), keys) / 16.0, -1)
    want = torch.einsum("ht,thd->hd", p, values).to(torch.bfloat16) * torch.sigmoid(qg[:, d:])
    dev = [t.to(cuda_device) for t in (qg, k_new, v_new, q_norm, k_norm)]
    for splits, device_position in ((1, False), (5, True), (74, False)):
        k, v = kc.to(cuda_device), vc.to(cuda_device)
        out = torch.empty(hq, d, dtype=torch.bfloat16, device=cuda_device)
        scratch = torch.full((lib().qd_attn_scratch_floats(hq, hk, d, splits),), float("nan"), device=cuda_device)
        counters = torch.zeros(hk, dtype=torch.int32, device=cuda_device)
        at = torch.tensor(position, dtype=torch.int32, device=cuda_device)
        for _ in range(2):                 # the counters are left ready for the next call
            call("qd_attn_decode", *map(ptr, dev), ptr(k), ptr(v), ptr(out), ptr(scratch), ptr(counters),
                 ptr(at) if device_position else None, 0 if device_position else position, cap, hq, hk, d, rotary, theta, eps,
                 splits, 0, stream_of(out))
        torch.testing.assert_close(out.cpu().float(), want.float(), rtol=2 ** -7, atol=2 ** -8 * float(want.float().abs().max()))
        torch.testing.assert_close(k[position].cpu().float(), wk[position].float(), rtol=2 ** -7, atol=1e-2)
        assert torch.equal(v[position].cpu(), v_new) and int(counters.sum()) == 0


# ----------------------------------------------------- the reference's saved fixtures
def test_reference_fixtures_through_the_operator_table(K, cuda_device, reference_fixtures):
    """The 15 saved block/step fixtures (tiny shapes, FP8 mixer projections) through
    bind_kernels(): output and post-call state within the stored tolerances."""
    from dataclasses import fields, is_dataclass
    table = K.bind_kernels()

    def compare(a, e, rtol, atol):
        if isinstance(e, torch.Tensor):
            if e.is_floating_point():
                torch.testing.assert_close(a.double().cpu(), e.double().cpu(), rtol=rtol, atol=atol)
            else:
                assert torch.equal(a.cpu(), e.cpu())
        elif is_dataclass(e):
            for f in fields(e):
                compare(getattr(a, f.name), getattr(e, f.name), rtol, atol)
        elif isinstance(e, (list, tuple)):
            for x, y in zip(a, e):
                compare(x, y, rtol, atol)
        elif isinstance(e, dict):
            for key in e:
                compare(a[key], e[key], rtol, atol)
        else:
            assert a == e

    state_args = {"full_attention_block": ("kv_cache",), "gated_delta_net_block": ("rec_state", "conv_state"),
                  "forward_step": ("state",)}
    for name, tree in sorted(reference_fixtures.items()):
        data = from_tree(tree, cuda_device)
        fn = data["function"]
        kwargs = data["kwargs"]
        actual = table[fn](**kwargs)
        compare(actual, data["expected"], data["rtol"], data["atol"])
        for arg in state_args.get(fn, ()):
            compare(kwargs[arg], data["after"][arg], data["rtol"], data["atol"])


@pytest.mark.parametrize("rows0,rows1,width", [(1, 1, 8), (32, 32, 2048), (256, 1, 2048), (7, 3, 2056), (5, 9, 2047), (9, 0, 4104)])
def test_bf16_matrices_of_one_input_share_a_launch(cuda_device, rows0, rows1, width):
    """Whole batches of 16-byte pieces, remainders and odd widths; bound: fp32 sums, one bf16 rounding (2^-8)."""
    from quickdraw_b200._lib import call, ptr, stream_of
    gen = torch.Generator(device=cuda_device).manual_seed(rows0)
    new = lambda *shape: torch.randn(shape, generator=gen, device=cuda_device).bfloat16()
    x, w0, w1 = new(width), new(rows0, width), new(rows1, width)
    y0, y1 = x.new_empty(rows0), x.new_empty(rows1)
    call("qd_bf16_gemv2", ptr(x), ptr(w0), ptr(y0), rows0, ptr(w1) if rows1 else None, ptr(y1) if rows1 else None, rows1, width, stream_of(x))
    for w, y in ((w0, y0), (w1, y1)):
        if w.shape[0]:
            want = w.double() @ x.double()
            torch.testing.assert_close(y.double(), want, rtol=2 ** -8, atol=1e-5 * float(want.abs().max()))


@pytest.mark.parametrize("rows", [1024, 333])                # a row count for the FP4 tensor core and one for the streaming kernel
@pytest.mark.parametrize("use", ["gate_up", "gemv", "gemv_streamed", "matmul_rows"])
def test_weights_written_right_in_front_of_their_use(K, cuda_device, use, rows):
    """Codes and scales that kernels of the same stream write, used at once, in buffers that held other matrices before: the
    same bits as behind a synchronisation."""
    if use == "matmul_rows":
        rows = 1024
    gen = torch.Generator(device=cuda_device).manual_seed(rows)
    new = lambda *shape: torch.randn(shape, generator=gen, device=cuda_device).bfloat16()
    a, b = new(4096, 4096), new(4096, 4096)
    x, chunk = new(2048), new(8, 2048)

    def product(gate, up):
        if use == "gate_up":
            return K.gate_up(x, gate, up)
        if use == "matmul_rows":
            return K.matmul_rows(chunk, up)[0]
        return K.nvfp4_gemv(x, up, force_generic=2 if use == "gemv_streamed" else False)

    got, projections = [], []
    for i in range(24):
        matrices = new(2, rows, 2048) * 2.0 ** (i % 5)
        torch.cuda.synchronize()
        if i % 3 == 0:
            torch.matmul(a, b)                                  # some hundred microseconds that everything below is queued behind
        projections.append([NVFP4Linear(*K.quantize_act(m)) for m in matrices])
        got.append(product(*projections[-1]))
        if i >= 8:                                              # their memory goes to a later matrix
            projections[i - 8] = [NVFP4Linear(p.weight.clone(), p.weight_scale.clone(), p.weight_scale_2.clone()) for p in projections[i - 8]]
    torch.cuda.synchronize()
    for pair, y in zip(projections, got):
        want = product(*pair)
        torch.cuda.synchronize()
        assert torch.equal(y, want)


@pytest.mark.parametrize("position", [999, 8191])
def test_decode_attention_keeps_its_probabilities_whole(cuda_device, position):
    """Head dimension 256, gates of one: fp32 probabilities and sums (2^-22 of the result) round 2^-22 / 2^-9 twice over, 2.4e-4, of
    the results to the other bf16 neighbour; probabilities of sixteen bits about 2e-3 of them."""
    from quickdraw_b200._lib import call, lib, ptr, stream_of
    differ = total = 0
    for seed in range(12):
        gen = torch.Generator(device=cuda_device).manual_seed(seed)
        new = lambda *shape: torch.randn(shape, generator=gen, device=cuda_device).bfloat16()
        keys, values = new(position + 1, 2, 256), new(position + 1, 2, 256)
        qg, k_new, v_new, norm = new(16, 2, 256), new(2, 256), new(2, 256), torch.zeros(256, dtype=torch.bfloat16, device=cuda_device)
        qg[:, 1] = 30.0
        out, counters = new(16, 256), torch.zeros(2, dtype=torch.int32, device=cuda_device)
        scratch = torch.empty(lib().qd_attn_scratch_floats(16, 2, 256, 74), device=cuda_device)
        call("qd_attn_decode", ptr(qg), ptr(k_new), ptr(v_new), ptr(norm), ptr(norm), ptr(keys), ptr(values), ptr(out), ptr(scratch), ptr(counters),
             None, position, position + 1, 16, 2, 256, 0, 1e6, 1e-6, 74, 0, stream_of(out))
        q = qg[:, 0].float()
        q = (q * torch.rsqrt(q.square().sum(-1, keepdim=True) / 256 + 1e-6)).bfloat16().double()
        k, v = (t.double().repeat_interleave(8, 1) for t in (keys, values))
        want = torch.einsum("ht,thd->hd", torch.softmax(torch.einsum("hd,thd->ht", q, k) / 16, -1), v)
        differ, total = differ + int((out != want.bfloat16()).sum()), total + out.numel()
    assert differ < total * 2 ** -10, differ / total


@pytest.mark.parametrize("position", [0, 20, 300])
def test_an_infinite_value_of_the_new_token_stays_infinite(cuda_device, position):
    """The last chunk of sixteen positions is not full: what its empty places multiply must not be the last row again."""
    from quickdraw_b200._lib import call, lib, ptr, stream_of
    gen = torch.Generator(device=cuda_device).manual_seed(position)
    new = lambda *shape: torch.randn(shape, generator=gen, device=cuda_device).bfloat16()
    keys, values, qg, k_new, v_new = new(position + 1, 2, 256), new(position + 1, 2, 256), new(16, 512), new(2, 256), new(2, 256)
    v_new[0, 7], v_new[1, 100] = float("inf"), float("-inf")
    norm, out, counters = torch.zeros(256, dtype=torch.bfloat16, device=cuda_device), new(16, 256), torch.zeros(2, dtype=torch.int32, device=cuda_device)
    scratch = torch.empty(lib().qd_attn_scratch_floats(16, 2, 256, 74), device=cuda_device)
    call("qd_attn_decode", ptr(qg), ptr(k_new), ptr(v_new), ptr(norm), ptr(norm), ptr(keys), ptr(values), ptr(out), ptr(scratch), ptr(counters),
         None, position, position + 1, 16, 2, 256, 64, 1e6, 1e-6, 74, 0, stream_of(out))
    infinite = torch.zeros(16, 256, dtype=torch.bool, device=cuda_device)
    infinite[:8, 7] = infinite[8:, 100] = True
    assert bool((out[:8, 7] == float("inf")).all()) and bool((out[8:, 100] == float("-inf")).all())
    assert bool(out[~infinite].isfinite().all())
