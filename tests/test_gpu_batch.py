"""Small-batch decode with per-sequence state against independent single-sequence runs (the
reference has no batched decode; its single-sequence step, applied to every sequence on its
own, is the oracle)."""

import math

import pytest
import torch

from oracle import decode_oracle as O
from quickdraw_b200 import synthetic

pytestmark = pytest.mark.gpu


def test_batched_state_kernels_equal_single_sequence_kernels(cuda_device):
    """Convolution and attention bit for bit, recurrence up to summation order, for sequences
    at different positions."""
    from quickdraw_b200._lib import call, ptr, stream_of
    batch, hk, hv, dk, dv, width = 3, 2, 4, 128, 128, 4
    channels = 2 * hk * dk + hv * dv
    src = synthetic.Source(23, "cpu")
    dev = cuda_device
    mixed = src.normal("mixed", batch, channels).to(dev)
    taps = src.normal("taps", channels, width, std=0.5).to(dev)
    a, b = src.normal("a", batch, hv).to(dev), src.normal("b", batch, hv).to(dev)
    a_log, dt_bias = src.normal("alog", hv, std=0.5).to(dev), src.normal("dt", hv).to(dev)
    conv0 = src.normal("conv0", batch, 2, channels, width - 1).to(dev)          # [batch, layers, ...]
    rec0 = src.normal("rec0", batch, 2, hv, dk, dv, std=0.1).float().to(dev)
    s = stream_of(mixed)
    layer = 1
    conv_b, rec_b = conv0.clone(), rec0.clone()
    conv_out, core = torch.empty_like(mixed), torch.empty(batch, hv * dv, dtype=torch.bfloat16, device=dev)
    call("qd_batch_gdn_conv", ptr(mixed), ptr(taps), ptr(conv_b[0, layer]), conv_b.stride(0), ptr(conv_out), batch,
         channels, width, s)
    call("qd_batch_gdn_recurrence", ptr(conv_out), ptr(a), ptr(b), ptr(a_log), ptr(dt_bias), ptr(rec_b[0, layer]),
         rec_b.stride(0), ptr(core), batch, hk, hv, dk, dv, s)
    conv_s, rec_s = conv0.clone(), rec0.clone()
    for i in range(batch):
        row, out = torch.empty(channels, dtype=torch.bfloat16, device=dev), torch.empty(hv * dv, dtype=torch.bfloat16, device=dev)
        call("qd_gdn_conv", ptr(mixed[i]), ptr(taps), ptr(conv_s[i, layer]), ptr(row), channels, width, s)
        call("qd_gdn_recurrence", ptr(row), ptr(a[i]), ptr(b[i]), ptr(a_log), ptr(dt_bias), ptr(rec_s[i, layer]), ptr(out),
             hk, hv, dk, dv, 0, s)
        torch.cuda.synchronize()
        assert torch.equal(row, conv_out[i])
        assert O.rel_l2(core[i].cpu(), out.cpu()) < 1e-2
    assert torch.equal(conv_b, conv_s)
    assert O.rel_l2(rec_b.cpu(), rec_s.cpu()) < 1e-4

    # attention: sequences at positions 0, 70, 300 of a 512-row cache
    hq, hkv, d, cap, splits = 8, 2, 256, 512, 8
    positions = torch.tensor([0, 70, 300], dtype=torch.int32, device=dev)
    qg = src.normal("qg", batch, hq, 2 * d).to(dev)
    k_new, v_new = src.normal("k", batch, hkv, d).to(dev), src.normal("v", batch, hkv, d).to(dev)
    q_norm, k_norm = src.normal("qn", d, std=0.1).to(dev), src.normal("kn", d, std=0.1).to(dev)
    k0, v0 = src.normal("kc", batch, 2, cap, hkv, d).to(dev), src.normal("vc", batch, 2, cap, hkv, d).to(dev)
    from quickdraw_b200._lib import lib
    floats = lib().qd_attn_scratch_floats(hq, hkv, d, splits)
    scratch = torch.empty(batch * floats, dtype=torch.float32, device=dev)
    counters = torch.zeros(batch * hkv, dtype=torch.int32, device=dev)
    kb, vb = k0.clone(), v0.clone()
    out_b = torch.empty(batch, hq * d, dtype=torch.bfloat16, device=dev)
    call("qd_batch_attn_decode", ptr(qg), ptr(k_new), ptr(v_new), ptr(q_norm), ptr(k_norm), ptr(kb[0, layer]),
         ptr(vb[0, layer]), kb.stride(0), ptr(out_b), ptr(scratch), ptr(counters), ptr(positions), batch, cap, hq, hkv,
         d, 64, 1e6, 1e-6, splits, s)
    ks, vs = k0.clone(), v0.clone()
    for i in range(batch):
        out = torch.empty(hq * d, dtype=torch.bfloat16, device=dev)
        call("qd_attn_decode", ptr(qg[i]), ptr(k_new[i]), ptr(v_new[i]), ptr(q_norm), ptr(k_norm), ptr(ks[i, layer]),
             ptr(vs[i, layer]), ptr(out), ptr(scratch), ptr(counters), None, int(positions[i]), cap, hq, hkv, d, 64,
             1e6, 1e-6, splits, 0, s)
        torch.cuda.synchronize()
        assert torch.equal(out, out_b[i]), (i, [O.rel_l2(out.float().cpu(), out_b[j].float().cpu()) for j in range(batch)])
    assert torch.equal(kb, ks) and torch.equal(vb, vs) and int(counters.abs().sum()) == 0

    # the lane-per-position form: same step up to summation order
    kl, vl = k0.clone(), v0.clone()
    out_l, q_scratch = torch.empty_like(out_b), torch.empty(batch, hq * d, dtype=torch.bfloat16, device=dev)
    for lane_splits in (8, 1):
        call("qd_batch_attention", ptr(qg), ptr(k_new), ptr(v_new), ptr(q_norm), ptr(k_norm), ptr(kl[0, layer]),
             ptr(vl[0, layer]), kl.stride(0), ptr(q_scratch), ptr(out_l), ptr(scratch), ptr(counters), ptr(positions),
             batch, cap, hq, hkv, d, 64, 1e6, 1e-6, lane_splits, s)
        torch.cuda.synchronize()
        for i in range(batch):
            assert O.rel_l2(out_l[i].float().cpu(), out_b[i].float().cpu()) < 1e-2, (lane_splits, i)
        assert O.rel_l2(kl.float().cpu(), kb.float().cpu()) < 1e-3 and torch.equal(vl, vb)
        assert int(counters.abs().sum()) == 0


def test_tall_projection_equals_row_by_row(cuda_device):
    from quickdraw_b200._lib import call, ptr, stream_of
    src = synthetic.Source(29, cuda_device)
    for tokens, rows, width in ((3, 40, 2048), (32, 257, 1024), (5, 4100, 2048), (33, 4096, 512), (32, 4112, 320), (200, 1, 2048), (130, 32, 2048), (64, 256, 2048), (70, 40, 192)):
        x, w = src.normal(f"x{tokens}", tokens, width), src.normal(f"w{rows}", rows, width, std=0.05)
        y = torch.empty(tokens, rows, dtype=torch.bfloat16, device=cuda_device)
        call("qd_seq_bf16_matmul", ptr(x), ptr(w), ptr(y), tokens, rows, width, stream_of(x))
        want = (x.double() @ w.double().T)
        assert O.rel_l2(y.cpu().double(), want.cpu()) < 4e-3
        # a second matrix of the same input in the same launch (or one after the other in the tall form): the same bits
        rows1 = 19
        w1 = src.normal(f"v{width}", rows1, width, std=0.05)
        y0, y1, alone = torch.empty_like(y), torch.empty(tokens, rows1, dtype=torch.bfloat16, device=cuda_device), None
        call("qd_seq_bf16_matmul2", ptr(x), ptr(w), ptr(y0), rows, ptr(w1), ptr(y1), rows1, tokens, width, stream_of(x))
        alone = torch.empty_like(y1)
        call("qd_seq_bf16_matmul", ptr(x), ptr(w1), ptr(alone), tokens, rows1, width, stream_of(x))
        assert torch.equal(y0, y) and torch.equal(y1, alone)


def test_batch_decode_follows_independent_sequences(cuda_device):
    """Three sequences with prompts of different lengths: every batched step's logits against
    the single-sequence step on a private copy of that sequence (same tokens fed to both)."""
    from quickdraw_b200.batch import BatchDecode, BatchState
    from quickdraw_b200.fused import FusedStep
    from quickdraw_b200.state import DecodeState
    cfg = synthetic.model_config(num_layers=4, vocab_size=4096, experts=16, topk=8)
    ckpt = synthetic.make_checkpoint(cfg, seed=5, device="cuda")
    single, batched = FusedStep(ckpt), BatchDecode(ckpt)
    lengths, steps, context = (5, 12, 20), 6, 64
    gen = torch.Generator().manual_seed(4)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=gen).to("cuda") for n in lengths]
    state = BatchState(cfg, len(lengths), context, "cuda")
    refs = []
    for b, prompt in enumerate(prompts):
        ref = DecodeState.allocate(cfg, context, "cuda")
        ref.kv_k.zero_()
        ref.kv_v.zero_()
        for position in range(len(prompt) - 1):
            single(ckpt, prompt[position], position, ref, logits=False)
        refs.append(ref)
        batched.run(prompt[:-1], 0, state.sequence(b))             # the single-sequence chunk prefill
        state.positions[b] = len(prompt) - 1
    tokens = torch.stack([p[-1] for p in prompts])
    errors = []
    for step in range(steps):
        want = [single(ckpt, tokens[b], lengths[b] - 1 + step, refs[b]).clone() for b in range(len(lengths))]
        picked, logits = batched.step(tokens, state)
        assert batched.check() == 0 and single.status() == 0
        for b in range(len(lengths)):
            errors.append(round(O.rel_l2(logits[b].float().cpu(), want[b].float().cpu()), 4))
            assert int(picked[b]) == int(logits[b].float().argmax())
        tokens = torch.stack([w.float().argmax() for w in want])
    # a step differs from the single-sequence step in summation order only; bf16 rounding points
    # amplify that to about 1e-2 on the logits, and a router near-tie that falls the other way
    # (one expert of eight exchanged for one token) to several times that; a flipped sequence
    # keeps the exchanged key/value rows for its remaining steps, so a third of the eighteen
    # comparisons may be off; the bulk is at the summation-order level
    assert sorted(errors)[len(errors) // 2] < 2e-2 and sorted(errors)[-7] < 3e-2 and max(errors) < 0.15, errors
    assert state.positions.tolist() == [n - 1 + steps for n in lengths]
    for b, ref in enumerate(refs):
        seq = state.sequence(b)
        n = lengths[b] - 1 + steps
        assert O.rel_l2(seq.rec_state.cpu(), ref.rec_state.cpu()) < 5e-2
        assert O.rel_l2(seq.conv_state.cpu(), ref.conv_state.cpu()) < 5e-2
        assert O.rel_l2(seq.kv_k[:, :n].cpu(), ref.kv_k[:, :n].cpu()) < 5e-2


def test_graph_replay_equals_eager_steps(cuda_device):
    """Five steps of four sequences issued launch by launch and replayed from the captured graph:
    same tokens, same logits, same state, bit for bit."""
    from quickdraw_b200.batch import BatchDecode, BatchState
    cfg = synthetic.model_config(num_layers=4, vocab_size=4096, experts=16, topk=8)
    ckpt = synthetic.make_checkpoint(cfg, seed=6, device="cuda")
    decoder = BatchDecode(ckpt)
    eager, replayed = BatchState(cfg, 4, 32, "cuda"), BatchState(cfg, 4, 32, "cuda")
    for state in (eager, replayed):
        state.positions.copy_(torch.tensor([0, 3, 7, 1], dtype=torch.int32))
    gen = torch.Generator().manual_seed(8)
    first = torch.randint(0, cfg.vocab_size, (4,), generator=gen).to("cuda")
    fed_a, fed_b = first.clone(), first.clone()
    for step in range(5):
        fed_a, logits_a = decoder.step(fed_a, eager)
        fed_b, logits_b = decoder.graph_step(fed_b, replayed)
        assert torch.equal(fed_a, fed_b) and torch.equal(logits_a, logits_b), step
        fed_b = fed_b.clone()
    assert decoder.check() == 0
    assert decoder._graphs[id(replayed)]["graph"] is not None
    assert eager.positions.tolist() == replayed.positions.tolist() == [5, 8, 12, 6]
    for name in ("kv_k", "kv_v", "rec_state", "conv_state"):
        assert torch.equal(getattr(eager, name), getattr(replayed, name)), name


def test_replay_of_a_small_state_after_a_larger_batch(cuda_device):
    """A state of two sequences is captured, another of 24 takes a step (which needs larger scratch), tensors are made where freed
    scratch could lie, then the first one's graph is replayed: as the eager steps of the same two sequences, bit for bit.  Contexts of 600
    positions, so that several blocks share a sequence and the counters decide who merges."""
    from quickdraw_b200.batch import BatchDecode, BatchState
    cfg = synthetic.model_config(num_layers=4, vocab_size=4096, experts=16, topk=8)
    decoder = BatchDecode(synthetic.make_checkpoint(cfg, seed=6, device="cuda"))
    eager, replayed, large = BatchState(cfg, 2, 640, "cuda"), BatchState(cfg, 2, 640, "cuda"), BatchState(cfg, 24, 640, "cuda")
    gen = torch.Generator(device="cuda").manual_seed(9)
    for name in ("kv_k", "kv_v", "rec_state", "conv_state"):
        getattr(eager, name).normal_(generator=gen).mul_(0.1)
        getattr(replayed, name).copy_(getattr(eager, name))
    for state in (eager, replayed):
        state.positions.copy_(torch.tensor([600, 517], dtype=torch.int32))
    fed_a = fed_b = torch.tensor([5, 77], device="cuda")
    kept = []
    for step in range(6):
        if step == 3:
            assert decoder._graphs[id(replayed)]["graph"] is not None
            decoder.step(torch.arange(24, device="cuda"), large)
            kept = [torch.full((n,), 3, dtype=torch.int32, device="cuda") for n in [1 << 8] * 64 + [1 << 18] * 4]
        fed_b, logits_b = (t.clone() for t in decoder.graph_step(fed_b, replayed))
        fed_a, logits_a = BatchDecode.step(decoder, fed_a, eager)
        assert torch.equal(fed_a, fed_b) and torch.equal(logits_a, logits_b), step
    assert all(bool((t == 3).all()) for t in kept) and decoder.check() == 0


@pytest.mark.parametrize("hq,hkv,d", [(16, 2, 256), (8, 2, 128)])
def test_batch_attention_forms_against_the_single_sequence_kernel(cuda_device, hq, hkv, d):
    """``qd_batch_attention`` (head dimension 256: tensor-core form with a full group of eight
    heads; 128: lane-per-position form) against the single-sequence decode attention, for
    sequences whose contexts end inside the first chunk, on a chunk boundary and deep in the cache."""
    from quickdraw_b200._lib import call, lib, ptr, stream_of
    dev, cap = cuda_device, 1024
    src = synthetic.Source(41, "cpu")
    positions = torch.tensor([0, 15, 16, 700, 1023], dtype=torch.int32, device=dev)
    batch = positions.numel()
    qg = src.normal("qg", batch, hq, 2 * d).to(dev)
    k_new, v_new = src.normal("k", batch, hkv, d).to(dev), src.normal("v", batch, hkv, d).to(dev)
    q_norm, k_norm = src.normal("qn", d, std=0.1).to(dev), src.normal("kn", d, std=0.1).to(dev)
    k0, v0 = src.normal("kc", batch, cap, hkv, d).to(dev), src.normal("vc", batch, cap, hkv, d).to(dev)
    floats = lib().qd_attn_scratch_floats(hq, hkv, d, 16)
    scratch = torch.empty(batch * floats, dtype=torch.float32, device=dev)
    counters = torch.zeros(batch * hkv, dtype=torch.int32, device=dev)
    s = stream_of(qg)
    ks, vs, want = k0.clone(), v0.clone(), []
    for i in range(batch):
        out = torch.empty(hq * d, dtype=torch.bfloat16, device=dev)
        call("qd_attn_decode", ptr(qg[i]), ptr(k_new[i]), ptr(v_new[i]), ptr(q_norm), ptr(k_norm), ptr(ks[i]), ptr(vs[i]),
             ptr(out), ptr(scratch), ptr(counters), None, int(positions[i]), cap, hq, hkv, d, 64, 1e6, 1e-6, 4, 0, s)
        want.append(out)
    for splits in (1, 5, 16):
        kb, vb = k0.clone(), v0.clone()
        # rows past every sequence's position are never read: poison them
        for i in range(batch):
            kb[i, int(positions[i]) + 1:] = float("nan")
            vb[i, int(positions[i]) + 1:] = float("nan")
        out_b, q_scratch = torch.empty(batch, hq * d, dtype=torch.bfloat16, device=dev), torch.empty(batch, hq * d, dtype=torch.bfloat16, device=dev)
        call("qd_batch_attention", ptr(qg), ptr(k_new), ptr(v_new), ptr(q_norm), ptr(k_norm), ptr(kb[0]), ptr(vb[0]),
             kb.stride(0), ptr(q_scratch), ptr(out_b), ptr(scratch), ptr(counters), ptr(positions), batch, cap, hq, hkv, d,
             64, 1e6, 1e-6, splits, s)
        torch.cuda.synchronize()
        assert int(counters.abs().sum()) == 0
        for i in range(batch):
            assert O.rel_l2(out_b[i].float().cpu(), want[i].float().cpu()) < 1e-2, (splits, i)
            n = int(positions[i]) + 1
            assert O.rel_l2(kb[i, :n].float().cpu(), ks[i, :n].float().cpu()) < 1e-3 and torch.equal(vb[i, :n], vs[i, :n])


@pytest.mark.parametrize("hq,hkv,lengths", [(16, 2, [1, 1024, 0, 33, 32, 1025, 31, 640]), (6, 3, [5]), (8, 1, [1000] * 40), (4, 2, list(range(1, 200))), (16, 2, [900] + [3] * 60)])
def test_batch_attention_shares_the_context_out(cuda_device, hq, hkv, lengths):
    """Blocks with parts of several sequences and sequences in several blocks, against the form with a block for each (sequence, KV head)
    (split count 1).  Lengths outside the cache (0, 1025) leave the output alone.  fp32 sums in another order, two bf16 roundings: 2^-7 of the largest."""
    from quickdraw_b200._lib import call, lib, ptr, stream_of
    dev, cap, d, batch = cuda_device, 1024, 256, len(lengths)
    gen = torch.Generator(device=dev).manual_seed(batch)
    new = lambda *shape: torch.randn(shape, generator=gen, device=dev).to(torch.bfloat16)
    qg, k_new, v_new, q_norm, k_norm = new(batch, hq * 2 * d), new(batch, hkv * d), new(batch, hkv * d), new(d) * 0.1, new(d) * 0.1
    k0, v0 = new(batch, cap, hkv, d), new(batch, cap, hkv, d)
    positions = torch.tensor(lengths, dtype=torch.int32, device=dev) - 1
    scratch = torch.empty(batch * lib().qd_attn_scratch_floats(hq, hkv, d, 16), device=dev)
    counters = torch.zeros(batch * hkv, dtype=torch.int32, device=dev)
    outs = []
    for splits in (1, 2, 3, 16):
        kb, vb = k0.clone(), v0.clone()
        for i, n in enumerate(lengths):
            kb[i, max(0, n):], vb[i, max(0, n):] = float("nan"), float("nan")
        out, q_scratch = torch.full((batch, hq * d), 7.0, dtype=torch.bfloat16, device=dev), torch.empty(batch, hq * d, dtype=torch.bfloat16, device=dev)
        call("qd_batch_attention", ptr(qg), ptr(k_new), ptr(v_new), ptr(q_norm), ptr(k_norm), ptr(kb), ptr(vb), kb.stride(0), ptr(q_scratch), ptr(out),
             ptr(scratch), ptr(counters), ptr(positions), batch, cap, hq, hkv, d, 64, 1e6, 1e-6, splits, stream_of(qg))
        assert int(counters.abs().sum()) == 0
        outs.append(out.float())
    outside = (positions < 0) | (positions >= cap)
    for out in outs:
        assert bool((out[outside] == 7.0).all()) and torch.isfinite(out).all()
        assert float((out - outs[0]).abs().max()) <= 2.0 ** -7 * float(outs[0][~outside].abs().max())


@pytest.mark.parametrize("hq,hkv,batch,length", [(16, 2, 8, 1000), (16, 2, 32, 1024), (4, 2, 60, 700), (8, 1, 3, 513), (8, 1, 200, 70)])
def test_batch_attention_of_a_sequence_does_not_depend_on_its_neighbours(cuda_device, hq, hkv, batch, length):
    """The same sequence in every place of a batch, beside neighbours of other lengths, some outside the cache: the same bits."""
    from quickdraw_b200._lib import call, lib, ptr, stream_of
    dev, cap, d = cuda_device, 1024, 256
    gen = torch.Generator(device=dev).manual_seed(length)
    new = lambda *shape: torch.randn(shape, generator=gen, device=dev).to(torch.bfloat16)
    qg, k_new, v_new, q_norm, k_norm = (new(1, n).expand(batch, n).contiguous() for n in (hq * 2 * d, hkv * d, hkv * d, d, d))
    k0, v0 = new(1, cap, hkv, d), new(1, cap, hkv, d)
    scratch = torch.empty(batch * lib().qd_attn_scratch_floats(hq, hkv, d, 16), device=dev)
    counters = torch.zeros(batch * hkv, dtype=torch.int32, device=dev)
    mine = torch.zeros(batch, dtype=torch.bool, device=dev)
    mine[0] = mine[batch // 2] = mine[-1] = True
    outs = []
    for others in ("same", 0, 1, 40, cap, cap + 1, "mixed"):
        lengths = torch.full((batch,), length, dtype=torch.int32, device=dev)
        if others == "mixed":
            lengths = torch.where(mine, lengths, torch.randint(0, cap + 2, (batch,), generator=gen, device=dev, dtype=torch.int32))
        elif others != "same":
            lengths[~mine] = others
        kb, vb = k0.expand(batch, -1, -1, -1).clone(), v0.expand(batch, -1, -1, -1).clone()
        out, q_scratch = (torch.full((batch, hq * d), 7.0, dtype=torch.bfloat16, device=dev) for _ in range(2))
        call("qd_batch_attention", ptr(qg), ptr(k_new), ptr(v_new), ptr(q_norm[0]), ptr(k_norm[0]), ptr(kb), ptr(vb), kb.stride(0), ptr(q_scratch),
             ptr(out), ptr(scratch), ptr(counters), ptr(lengths - 1), batch, cap, hq, hkv, d, 64, 1e6, 1e-6, 16, stream_of(qg))
        assert int(counters.abs().sum()) == 0
        outs += [out[i] for i in range(batch) if mine[i]]
    assert torch.isfinite(outs[0]).all() and all(torch.equal(o, outs[0]) for o in outs)


def test_batch_decode_with_the_published_checkpoint_formats(cuda_device):
    """FP8 mixers and an NVFP4 LM head in the batched step (E4M3 x E4M3 product, NVFP4 rows form):
    the first step of two sequences from empty state against the single-sequence step (one step:
    E4M3 rounding steps and router ties do not propagate)."""
    from quickdraw_b200.batch import BatchDecode, BatchState
    from quickdraw_b200.fused import FusedStep
    from quickdraw_b200.state import DecodeState
    cfg = synthetic.model_config(num_layers=2, vocab_size=2048, experts=16, topk=8, interval=2)     # one DeltaNet, one attention layer
    ckpt = synthetic.make_checkpoint(cfg, seed=21, device="cuda", fp8_mixers=True, nvfp4_head=True)
    single, batched = FusedStep(ckpt), BatchDecode(ckpt)
    state = BatchState(cfg, 2, 16, "cuda")
    tokens = torch.tensor([17, 1200], device="cuda")
    picked, logits = batched.step(tokens, state)
    assert batched.check() == 0
    for b in range(2):
        ref = DecodeState.allocate(cfg, 16, "cuda")
        for t in (ref.kv_k, ref.kv_v, ref.rec_state, ref.conv_state):
            t.zero_()
        want = single(ckpt, tokens[b], 0, ref)
        assert O.rel_l2(logits[b].float().cpu(), want.float().cpu()) < 5e-2, b
        seq = state.sequence(b)
        assert O.rel_l2(seq.rec_state.cpu(), ref.rec_state.cpu()) < 1e-2 and O.rel_l2(seq.conv_state.cpu(), ref.conv_state.cpu()) < 1e-3
    assert single.status() == 0


@pytest.mark.parametrize("batch,hk,hv,dv", [(1, 1, 1, 128), (5, 2, 6, 128), (3, 1, 2, 20), (2, 2, 2, 260), (3, 1, 2, 18)])
def test_batch_recurrence_equals_the_sequences_one_by_one(cuda_device, batch, hk, hv, dv):
    """One token of every sequence (a block of whole rows of the state; 18 columns: the kernel for runs) against the run kernel on each sequence alone.
    fp32 sums of 128 terms in another order: 2^-18 of the state, one bf16 rounding of the results."""
    from quickdraw_b200._lib import call, ptr, stream_of
    gen = torch.Generator(device=cuda_device).manual_seed(batch + dv)
    new = lambda *shape: torch.randn(shape, generator=gen, device=cuda_device).to(torch.bfloat16)
    qkv, a, b, a_log, bias = new(batch, 2 * hk * 128 + hv * dv), new(batch, hv), new(batch, hv), new(hv), new(hv)
    state = torch.randn(batch, hv, 128, dv, generator=gen, device=cuda_device)
    one, out, alone = state.clone(), torch.full((batch, hv * dv), float("nan"), dtype=torch.bfloat16, device=cuda_device), torch.empty(batch, hv * dv, dtype=torch.bfloat16, device=cuda_device)
    call("qd_batch_gdn_recurrence", ptr(qkv), ptr(a), ptr(b), ptr(a_log), ptr(bias), ptr(state), state.stride(0), ptr(out), batch, hk, hv, 128, dv, stream_of(qkv))
    for z in range(batch):
        call("qd_seq_gdn_recurrence", ptr(qkv[z]), ptr(a[z]), ptr(b[z]), ptr(a_log), ptr(bias), ptr(one[z]), ptr(alone[z]), 1, hk, hv, 128, dv, stream_of(qkv))
    assert float((state - one).abs().max()) <= 2.0 ** -18 * float(one.abs().max())
    assert float((out.double() - alone.double()).abs().max()) <= 2.0 ** -8 * float(alone.double().abs().max())


@pytest.mark.parametrize("rows,columns,kind", [(32, 151936, "plain"), (3, 1000, "ties"), (1, 7, "plain"), (5, 4099, "negative"), (4, 33000, "nan"), (2, 16, "zeros"), (2, 264, "lowest")])
def test_argmax_of_rows(cuda_device, rows, columns, kind):
    """The greedy choice as torch makes it of the same values in fp32: the first of equal ones, -0 equal to 0, NaN above infinity."""
    from quickdraw_b200._lib import call, ptr, stream_of
    gen = torch.Generator(device=cuda_device).manual_seed(columns)
    x = torch.randn(rows, columns, generator=gen, device=cuda_device)
    x = {"ties": x.round(), "negative": -x.abs() - 1, "zeros": torch.zeros_like(x) * (x - 1).sign(), "lowest": torch.full_like(x, -math.inf)}.get(kind, x).to(torch.bfloat16)
    if kind == "nan":
        x[1, 5], x[1, 20000], x[1, 31000], x[2, 32999] = math.inf, math.nan, math.nan, math.inf
    picked = torch.full((rows,), -1, dtype=torch.long, device=cuda_device)
    call("qd_argmax_rows", ptr(x), rows, columns, ptr(picked), stream_of(x))
    values = x.float().nan_to_num(nan=math.inf, posinf=3e38).cpu()
    first = torch.where(values == values.amax(1, keepdim=True), torch.arange(columns), columns).amin(1)
    assert picked.tolist() == first.tolist()
