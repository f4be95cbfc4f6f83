"""Host-side logic that needs no GPU: the C-ABI library loads and exports every symbol the
header declares, a missing library fails loudly (there is no fallback path), and the engine's
request control flow (reference behaviour: quickdraw/engine/engine.py:93-148, exercised the way
tests/engine/test_engine.py of the reference does, with an injected step)."""

import re
from pathlib import Path

import pytest
import torch

from quickdraw_b200 import _lib, synthetic
from quickdraw_b200.engine import Engine
from quickdraw_b200.weights import Checkpoint

ROOT = Path(__file__).resolve().parents[1]
HEADER = ROOT / "include" / "quickdraw_b200.h"


def declared_symbols() -> list[str]:
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return sorted(set(re.findall(r"\b(qd_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    names = declared_symbols()
    assert len(names) >= 30 and "qd_decode_step_persistent" in names and "qd_attn_decode_static" in names
    handle = _lib.lib()
    for name in names:
        assert hasattr(handle, name), f"{name} is declared in the header but not exported"
    assert handle.qd_version() >= 1
    assert handle.qd_error_string(3) == b"bounded device wait ran out"


def test_binding_table_covers_the_header():
    assert set(declared_symbols()) == set(_lib.exported_symbols())


def test_binding_argument_types_follow_the_header():
    """Every ctypes signature has the header's parameters, in order: pointers, int, unsigned, float, long long."""
    import ctypes
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    kinds = {ctypes.c_void_p: "pointer", ctypes.c_int: "int", ctypes.c_float: "float", ctypes.c_longlong: "long long",
             ctypes.c_uint: "unsigned int"}
    checked = 0
    for result, name, params in re.findall(r"\b(int|long long|const char\*)\s+(qd_[a-z0-9_]+)\s*\(([^)]*)\)\s*;", text):
        if name == "qd_error_string":
            continue
        declared = []
        for param in (piece.strip() for piece in params.split(",")):
            if param in ("", "void"):
                continue
            if "*" in param:
                declared.append("pointer")
            else:
                declared.append(re.sub(r"\s+\w+$", "", param).replace("const ", "").strip())
        bound = [kinds[t] for t in _lib.SIGNATURES[name]]
        assert bound == declared, (name, bound, declared)
        assert (name in _lib.LONG_RESULTS) == (result == "long long"), name
        checked += 1
    assert checked == len(_lib.SIGNATURES)


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "libquickdraw_b200.so")
    with pytest.raises(_lib.LibraryMissing, match="no fallback"):
        _lib.lib()
    from quickdraw_b200 import kernels
    x = torch.zeros(2048, dtype=torch.bfloat16)
    with pytest.raises((_lib.LibraryMissing, AssertionError)):
        kernels.rms_norm(x, torch.ones(2048), 1e-6)


# ------------------------------------------------------------------------- engine control flow
class CountingStep:
    """A step that emits a fixed token sequence: logits peak at script[position]."""

    def __init__(self, vocab, script):
        self.vocab, self.script, self.calls = vocab, script, []

    def __call__(self, ckpt, token_id, position, state, **kwargs):
        self.calls.append((int(token_id), int(position)))
        state.rec_state.add_(1.0)
        logits = torch.zeros(self.vocab)
        logits[self.script[int(position) % len(self.script)]] = 1.0
        return logits


def make_engine(script, max_context=16):
    cfg = synthetic.model_config(num_layers=4, vocab_size=64)
    ckpt = Checkpoint(config=cfg, embed_tokens=None, final_norm=None, lm_head=None, layers=[])
    step = CountingStep(cfg.vocab_size, script)
    return Engine(ckpt, max_context=max_context, device="cpu", step=step), step


def test_custom_step_selects_custom_backend_without_graph():
    engine, _ = make_engine([1])
    assert engine.backend == "custom" and engine.graph is None and engine.state.position == 0


def test_b200_backend_refuses_a_cpu_device():
    cfg = synthetic.model_config(num_layers=4, vocab_size=64)
    ckpt = Checkpoint(config=cfg, embed_tokens=None, final_norm=None, lm_head=None, layers=[])
    with pytest.raises(AssertionError, match="no CPU path"):
        Engine(ckpt, max_context=8, device="cpu")


def test_generate_runs_the_prompt_once_then_decodes():
    engine, step = make_engine([3, 4, 5, 6, 7, 8, 9, 10])
    out = engine.generate([20, 21, 22], 4)
    # prompt tokens at positions 0..2; the logits after position 2 pick script[2] = 5; every
    # decode step feeds the previous choice at the next position
    assert out == [5, 6, 7, 8]
    assert step.calls == [(20, 0), (21, 1), (22, 2), (5, 3), (6, 4), (7, 5)]
    assert engine.state.position == 6


def test_generate_stops_at_eos_and_keeps_it():
    engine, _ = make_engine([3, 4, 5, 6, 7, 8])
    engine.eos_token_ids = {6}
    assert engine.generate([1, 2], 10) == [4, 5, 6]


def test_generate_stops_at_capacity():
    engine, _ = make_engine([1, 2, 3, 4, 5, 6, 7, 8], max_context=5)
    out = engine.generate([9, 9, 9], 10)
    assert len(out) == 3 and engine.state.position == 5       # prompt 3 + two decode steps fit


def test_generate_argument_contract():
    engine, step = make_engine([1])
    assert engine.generate([1, 2], 0) == [] and step.calls == []
    with pytest.raises(AssertionError, match="nonnegative"):
        engine.generate([1], -1)
    with pytest.raises(AssertionError, match="prompt must fit"):
        engine.prefill([])
    with pytest.raises(AssertionError, match="prompt must fit"):
        engine.prefill(list(range(17)))
    with pytest.raises(AssertionError, match="pending token"):
        engine.decode_step()


def test_reset_zeroes_history_and_keeps_the_buffers():
    engine, _ = make_engine([1, 2, 3])
    engine.generate([5, 6], 2)
    addresses = [t.data_ptr() for t in (engine.state.kv_k, engine.state.rec_state, engine.state.conv_state)]
    assert float(engine.state.rec_state.abs().sum()) > 0
    engine.reset()
    assert engine.state.position == 0 and engine.pending_token is None
    assert float(engine.state.rec_state.abs().sum()) == 0 and float(engine.state.conv_state.abs().sum()) == 0
    assert addresses == [t.data_ptr() for t in (engine.state.kv_k, engine.state.rec_state, engine.state.conv_state)]


def test_prefill_starts_a_fresh_request():
    engine, step = make_engine([1, 2, 3, 4])
    engine.generate([7, 7, 7], 1)
    engine.prefill([8])
    assert engine.state.position == 1 and step.calls[-1] == (8, 0)


# ----------------------------------------------------------------- conversation reuse (host logic)
def test_prefix_reuse_processes_only_the_new_suffix():
    engine, step = make_engine([3, 4, 5, 6, 7, 8, 9, 10], max_context=32)
    engine.prefill_reuse([20, 21, 22])
    assert engine.reused_tokens == 0 and [c for c in step.calls] == [(20, 0), (21, 1), (22, 2)]
    before = engine.state.rec_state.clone()
    step.calls.clear()
    logits = engine.prefill_reuse([20, 21, 22, 30, 31])                # extends the previous prompt
    assert engine.reused_tokens == 3 and step.calls == [(30, 3), (31, 4)]
    assert engine.state.position == 5 and int(logits.argmax()) == 7    # script[4]
    assert torch.equal(engine.state.rec_state, before + 2)             # restored, then two more steps
    step.calls.clear()
    engine.prefill_reuse([20, 21, 99, 30])                             # diverges inside the old prompt: fresh
    assert engine.reused_tokens == 0 and step.calls[0] == (20, 0) and len(step.calls) == 4
    assert torch.equal(engine.state.rec_state, torch.full_like(before, 4.0))


def test_snapshot_restore_round_trip_and_binding():
    engine, step = make_engine([3, 4, 5, 6, 7, 8, 9, 10], max_context=32)
    first = engine.generate([1, 2], 3)                                  # prompt 2 + decode steps at positions 2, 3
    snap = engine.snapshot()
    assert snap.tokens == (1, 2, first[0], first[1]) and snap.position == 4
    assert snap.nbytes() == engine.state.rec_state.nbytes + engine.state.conv_state.nbytes
    rec = engine.state.rec_state.clone()
    engine.decode_step()
    engine.decode_step()
    engine.restore(snap)                                                # back to the snapshot: buffers reused
    assert engine.state.position == 4 and torch.equal(engine.state.rec_state, rec)
    assert int(engine.pending_token) == first[2]
    assert int(engine.decode_step()) == 7                               # continues as it did the first time (script[4])
    # a new conversation overwrites the cache rows the snapshot relies on
    engine.prefill([9, 9, 9, 9, 9])
    with pytest.raises(AssertionError, match="overwritten"):
        engine.restore(snap)
    other, _ = make_engine([1], max_context=32)
    with pytest.raises(AssertionError, match="another checkpoint"):
        other.restore(snap)


def test_reuse_survives_a_reset_when_the_cache_rows_are_intact():
    engine, step = make_engine([3, 4, 5, 6], max_context=32)
    engine.prefill_reuse([5, 6, 7])
    engine.reset()                                                      # history cleared, cache rows untouched
    step.calls.clear()
    engine.prefill_reuse([5, 6, 7, 8])
    assert engine.reused_tokens == 3 and step.calls == [(8, 3)]


def test_bench_byte_counts_of_a_step_and_of_a_batched_step():
    """The algorithmic bytes bench.py divides by: one sequence of the batched count is the single-token
    count (up to the norm vectors and the embedding row), more sequences add their own state and KV
    history and touch more distinct experts, never more than all of them."""
    import importlib.util
    spec = importlib.util.spec_from_file_location("bench", Path(__file__).resolve().parents[1] / "bench.py")
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    cfg = synthetic.model_config()
    one, single = bench.bytes_per_batch_step(cfg, 1, 639), bench.bytes_per_token(cfg, 639)
    assert abs(one - single) < 1e-3 * single
    small, large = bench.bytes_per_batch_step(cfg, 32, 8192), bench.bytes_per_batch_step(cfg, 64, 8192)
    assert one < small < large
    # 32 more sequences: their state and KV history, and fewer than 32 x 8 more experts per layer
    h, inter = cfg.hidden_size, cfg.moe_intermediate_size
    expert = 3 * (inter * h // 2 + inter * h // 16 + 4)
    per_sequence = (large - small) / 32
    state = 36 * 2 * (32 * 128 * 128 * 4 + 8192 * 3 * 2) + 12 * 2 * 2 * 256 * 2 * 8193
    assert state < per_sequence < state + cfg.num_hidden_layers * 8 * expert


@pytest.mark.parametrize("tokens,fp8", [(3, False), (70, False), (3, True), (40, True)])
def test_chunk_and_batch_paths_pass_the_declared_number_of_arguments(monkeypatch, tokens, fp8):
    """The Python drivers of the prompt-chunk and batched-decode paths, run on CPU tensors with the library
    call replaced by a recorder: every call names a bound entry point and passes as many arguments as the
    header declares for it (ctypes would not notice a missing trailing argument), and both paths reach
    their few-row and many-row forms."""
    from quickdraw_b200 import batch, prefill
    from quickdraw_b200.state import DecodeState
    seen = {}

    def record(name, *args):
        assert name in _lib.SIGNATURES, name
        assert len(args) == len(_lib.SIGNATURES[name]), (name, len(args), len(_lib.SIGNATURES[name]))
        seen[name] = seen.get(name, 0) + 1

    class FakeLibrary:
        def __getattr__(self, name):
            assert name in _lib.SIGNATURES, name
            return lambda *args: 4096 if name.endswith("_bytes") else 1

    for module in (prefill, batch):
        monkeypatch.setattr(module, "call", record)
        monkeypatch.setattr(module, "lib", lambda: FakeLibrary())
        monkeypatch.setattr(module, "stream_of", lambda t: None)
    class AsIfOnGpu(torch.Tensor):         # the drivers refuse token ids that are not on a GPU
        is_cuda = property(lambda self: True)

    cfg = synthetic.model_config(num_layers=4, vocab_size=512, experts=16, topk=4)
    ckpt = synthetic.make_checkpoint(cfg, seed=2, device="cpu", fp8_mixers=fp8, nvfp4_head=fp8)
    state = DecodeState.allocate(cfg, 128, "cpu")
    prefill.ChunkPrefill(ckpt).run((torch.arange(tokens) % cfg.vocab_size).as_subclass(AsIfOnGpu), 0, state)
    assert seen.get("qd_seq_moe_combine_norm", 0) == 3 and "qd_seq_moe_combine" not in seen      # the last MoE block is not run
    assert ("qd_fp8_matmul" in seen) == fp8
    assert ("qd_nvfp4_expert_rows2" in seen) or ("qd_nvfp4_grouped_matmul" in seen)
    chunk_calls = dict(seen)
    seen.clear()
    many = batch.BatchState(cfg, 3, 64, "cpu")
    decoder = batch.BatchDecode(ckpt)
    monkeypatch.setattr(decoder, "_attn_splits", lambda *a: 1, raising=False)
    picked, logits = decoder.step(torch.tensor([1, 2, 3]).as_subclass(AsIfOnGpu), many)
    assert picked.shape == (3,) and logits.shape == (3, cfg.vocab_size) and many.positions.tolist() == [1, 1, 1]
    assert seen["qd_seq_moe_combine_norm"] == 4 and seen["qd_nvfp4_expert_rows2"] == 4 and seen["qd_seq_bf16_matmul2"] >= 4
    assert "qd_nvfp4_matmul_rows3" in seen or fp8
    assert chunk_calls


def test_every_kernel_launched_as_a_programmatic_dependent_waits_for_its_predecessor():
    """Source check: a kernel that qd_launch may start before the kernel in front of it has finished
    (pdl argument other than false / 0) contains the wait, as chain_enter() or grid_dependency_wait()."""
    sources = {path.name: path.read_text() for path in (ROOT / "quickdraw_b200" / "csrc").glob("*.cu*")}

    def arguments(text, start):          # top-level arguments of the call whose "(" ends at `start`
        depth, current, found, i = 0, "", [], start
        while True:
            ch = text[i]
            if ch in "([":
                depth += 1
            elif ch in ")]":
                if depth == 0:
                    return found + [current.strip()]
                depth -= 1
            if ch == "," and depth == 0 and (found or current.count("<") == current.count(">")):      # template arguments of the kernel
                found.append(current.strip())
                current = ""
            else:
                current += ch
            i += 1

    def bodies(kernel):
        for text in sources.values():
            for match in re.finditer(r"__global__[^{;]*?\b" + kernel + r"\s*\(", text, flags=re.S):
                start = text.index("{", match.end())
                depth, end = 0, start
                while True:
                    depth += {"{": 1, "}": -1}.get(text[end], 0)
                    if depth == 0:
                        break
                    end += 1
                yield text[start:end]

    dependents = 0
    for name, text in sources.items():
        for match in re.finditer(r"(?<!int )qd_launch\(", text):
            args = arguments(text, match.end())
            kernel, pdl = re.match(r"\w+", args[0]).group(0), args[5]
            if pdl in ("false", "0"):
                continue
            found = list(bodies(kernel))
            assert found, (name, kernel)
            assert all("chain_enter();" in body or "grid_dependency_wait();" in body for body in found), (name, kernel)
            dependents += 1
    assert dependents >= 30



def test_operator_table_kernels_read_nothing_before_their_wait():
    """Source check: what the operator table launches as a programmatic dependent (mode 3) may follow a kernel that writes any of
    its operands, weights included, so no operand is read in front of the wait; and the kernels whose results may be weights
    or states that others fetch ahead of their own wait release nobody before they end."""
    sources = {path.name: path.read_text() for path in (ROOT / "quickdraw_b200" / "csrc").glob("*.cu*")}
    everything = "\n".join(sources.values())

    def kernel(name):                    # (parameters, body)
        match = re.search(r"__global__[^{;]*?\b" + name + r"\s*\(([^{;]*)\)\s*\{", everything, flags=re.S)
        depth, at = 1, match.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(everything[at], 0)
            at += 1
        return match.group(1), re.sub(r"//[^\n]*", "", everything[match.end():at - 1])

    names = set(re.findall(r"qd_launch\((?:qd::)?(\w+)(?:<\w+>)?, (?:[^;]*?), 3, ", everything))
    names |= {"attn_decode_kernel", "attn_decode_mma_kernel", "moe_down_kernel"}          # the mode is an argument of their entry points
    assert names >= {"rms_norm_kernel", "add_norm_kernel", "bf16_gemv_kernel", "route_kernel", "act_quantize_kernel", "gdn_conv_kernel",
                     "nvfp4_umma_matvec_kernel", "nvfp4_gemm_w4a4_kernel"}
    waits = r"chain_enter\(\);|grid_dependency_wait\(\);"
    for name in names:
        parameters, body = kernel(name)
        front = body[:re.search(waits, body).start()]
        pointers = re.findall(r"\*\s*(?:const\s+)?(?:__restrict__\s+)?(\w+)", parameters)
        reads = [p for p in pointers if re.search(r"\b" + p + r"\s*\[|[=(,+]\s*\*" + p + r"\b", front)]
        assert not reads and not re.search(r"\bp\.\w+\s*\[|\*\s*p\.\w+\s*[;)]|\bld_\w+\(|\bload\w*\(|__ldc?g\(|bulk_load|cp16|copy16", front), (name, reads)
    _, body = kernel("stream_kernel")    # fetches weights ahead of the wait in the decode step, not here
    assert body.index("if (p.ids_in || p.wait_first) grid_dependency_wait();") < body.index("bulk_load(")
    entry = sources["stream.cu"][sources["stream.cu"].index("int qd_stream_matvec_try("):]
    assert entry.index("p.prologue = PRO_NONE;") < entry.index("p.wait_first = 1;") < entry.index("return stream_launch(p, 0, stream, 3);")
    for name in ("act_quantize_kernel", "nvfp4_gemm_w4a4_kernel", "w4a4_pair_kernel", "rms_norm_kernel", "gdn_conv_kernel"):
        body = kernel(name)[1]
        assert "chain_enter" not in body and "grid_launch_dependents" not in body, name


def test_tensor_memory_is_read_by_whole_warps():
    """Source check of the tcgen05 products of fp32 rows and of static FP8: the collective reads follow a wait whose result the warp
    shares, and no lane leaves an iteration (a token past the last one) on its own."""
    csrc = ROOT / "quickdraw_b200" / "csrc"
    for name, kernel, read in (("fp8_gemm.cu", "fp8_gemm_kernel", "tmem_load16("), ("linear.cu", "linear_pieces_kernel", "tmem_ld32(")):
        text = (csrc / name).read_text()
        body = text[re.search(r"\b" + kernel + r"\(const", text).start():]
        epilogue = body[body.rindex("const int ", 0, body.index(read)):body.index("__syncthreads();", body.index(read))]
        before = body[:body.index(read)]
        assert re.search(r"ok = __all_sync\(0xffffffffu, (?:ok && )?mbar_wait\(ready", before[before.rindex("} else {\n        const int "):]), name
        assert "continue;" not in epilogue, name


def test_a_wait_that_ran_out_leaves_nothing_in_flight():
    """Source check of the tcgen05 kernels with several warps of bounded waits: tensor memory is given back behind a commit of all
    MMAs, which no earlier result guards, and the attention's loaders wait for the copies they have started in any case."""
    csrc = ROOT / "quickdraw_b200" / "csrc"
    for name, kernel in (("fp8_gemm.cu", "fp8_gemm_kernel"), ("linear.cu", "linear_pieces_kernel"), ("flash_umma.cuh", "flash_umma_kernel"),
                         ("expert_tiles.cu", "expert_tiles_kernel"), ("gemm4.cu", "w4a4_pair_kernel"), ("linear_pair.cuh", "linear_pair_kernel")):
        text = (csrc / name).read_text()
        body = text[re.search(r"\b" + kernel + r"\(const", text).start():]
        body = body[:min(body.index(word) for word in ("tmem_dealloc", "tcgen05.dealloc") if word in body)]
        assert re.search(r"commit\w*\(&?(?:bars->)?drained\);[^\n]*\n\s*mbar_wait\(&?(?:bars->)?drained, 0", body), name
    for name, kernel in (("gemm4.cu", "w4a4_pair_kernel"), ("linear_pair.cuh", "linear_pair_kernel")):
        body = (csrc / name).read_text()
        body = body[re.search(r"\b" + kernel + r"\(const", body).start():]
        body = body[:body.index("pair_tmem_dealloc")]
        # pairs of blocks: the first one issues, and waits for the commit before the blocks meet; loads end when they are taken
        assert "\n        if (n) pair_loads_taken(" in body and "cluster_sync();" in body[body.index("drained, 0"):], name
    loaders = (csrc / "flash_umma.cuh").read_text()
    assert re.search(r"\n        if \(issued >= 0\) mbar_wait\(full, \(issued >> 1\) & 1, nullptr\);", loaders)


def test_another_block_is_known_to_run_before_its_memory_is_used():
    """Source check of the kernels that reach into another block's shared memory: a barrier of the whole cluster is waited for in front of
    the first such access (until then the other block may not have started)."""
    remote, waits = r"\bmapa\b|\bof_first_block\(|\bmap_shared_rank\(", r"\bcluster_sync\(\);|barrier\.cluster\.wait|\bbarrier_wait\(\);|\bcluster\.sync\(\);"
    found = set()
    for path in (ROOT / "quickdraw_b200" / "csrc").glob("*.cu*"):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for match in re.finditer(r"__global__[^{;]*?\b(\w+)\s*\((?:[^{;()]|\([^()]*\))*\)\s*\{", text, flags=re.S):
            depth, at = 1, match.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            body = text[match.end():at]
            access = re.search(remote, body)
            if access:
                found.add(match.group(1))
                wait = re.search(waits, body)
                assert wait and wait.start() < access.start(), (path.name, match.group(1))
    assert found >= {"argmax_rows_kernel", "linear_pair_kernel", "w4a4_pair_kernel", "recurrence_step_kernel"}, found


def test_a_stage_of_scales_belongs_to_one_group_of_warps():
    """Source check of the FP4 product on pairs of SMs: the groups that move block scales take every step once, and whoever waits for a
    stage of the ring has waited for each of its rounds before (the parity of a barrier tells neighbouring rounds apart, no more)."""
    text = (ROOT / "quickdraw_b200" / "csrc" / "gemm4.cu").read_text()
    stages, groups = (int(re.search(r"struct Pair4 \{.*?\b" + name + r" = (\d+)", text, flags=re.S).group(1)) for name in ("kStages", "kScaleGroups"))
    step = re.search(r"for \(int it = group; it < steps; it (\+?=) ([^)]*\)?)\) \{", text)
    if step.group(1) == "+=":
        after = lambda it: it + groups
    else:
        assert step.group(2) == "next_scale_step(it)"
        test, yes, no = re.search(r"int next_scale_step\(int it\) \{.*?return (.*?) \? (.*?) : (.*?);", text, flags=re.S).groups()
        after = eval(f"lambda it: ({yes}) if ({test}) else ({no})".replace("/", "//"), {"S": stages, "G": groups})
    owners, taken = {}, []
    for group in range(groups):
        it = group
        while it < 20 * stages * groups:
            owners.setdefault(it % stages, set()).add(group)
            taken.append(it)
            it = after(it)
    assert sorted(taken) == list(range(20 * stages * groups)) and all(len(who) == 1 for who in owners.values()), owners


def test_banks_off_a_16_byte_boundary_keep_the_form_that_takes_them():
    """The launch of gate, up and SwiGLU refuses such addresses, the grouped product does not: a chunk goes the second way then."""
    from types import SimpleNamespace

    from quickdraw_b200.prefill import ChunkPrefill
    from quickdraw_b200.weights import NVFP4Linear
    prefill = ChunkPrefill.__new__(ChunkPrefill)
    prefill.total_experts = 64

    def bank(rows, width, shift="", by=8):
        def part(name, *shape):
            count = torch.Size(shape).numel()
            flat = torch.zeros(count + by, dtype=torch.uint8)
            return (flat[by:] if name == shift else flat[:count]).view(shape)
        return NVFP4Linear(part("codes", 64, rows, width // 2), part("scales", 64, rows, width // 16), torch.ones(()))

    plain = {"experts_gate": bank(512, 256), "experts_up": bank(512, 256), "experts_down": bank(256, 512)}
    assert prefill._tiles_form(64 * 64, SimpleNamespace(**plain))
    for name, b in plain.items():
        for shift in ("codes", "scales"):
            assert not prefill._tiles_form(64 * 64, SimpleNamespace(**{**plain, name: bank(b.out_features, b.in_features, shift)})), (name, shift)


def test_small_expert_banks_keep_the_few_rows_form():
    """Where the launch of gate, up and SwiGLU was measured to be the slower one, and where it was the faster."""
    from types import SimpleNamespace

    from quickdraw_b200.prefill import ChunkPrefill
    from quickdraw_b200.weights import NVFP4Linear
    prefill = ChunkPrefill.__new__(ChunkPrefill)
    for experts, hidden, inner, slower, faster in ((16, 1024, 512, (6, 12, 20), (21, 200)), (16, 2048, 512, (8, 12), (24,)), (32, 2048, 512, (4, 6), (8, 40)),
                                                   (64, 2048, 512, (4, 6), (8, 20)), (256, 2048, 512, (4,), (6, 8, 64))):
        bank = lambda rows, width: NVFP4Linear(torch.empty(experts, rows, width // 2, dtype=torch.uint8),
                                               torch.empty(experts, rows, width // 16, dtype=torch.uint8), torch.ones(()))
        w = SimpleNamespace(experts_gate=bank(inner, hidden), experts_up=bank(inner, hidden), experts_down=bank(hidden, inner))
        prefill.total_experts = experts
        assert not any(prefill._tiles_form(n * experts, w) for n in slower), (experts, hidden)
        assert all(prefill._tiles_form(n * experts, w) for n in faster), (experts, hidden)


def test_launch_modes_of_the_entry_points():
    """Any value but 0 asked for a dependent launch before the third mode existed, and still does: no other value of a caller
    reaches the launch helper's modes of its own."""
    csrc = ROOT / "quickdraw_b200" / "csrc"
    assert "{ return pdl == 3 ? 3 : pdl != 0; }" in (csrc / "common.cuh").read_text()
    for name in ("attention.cu", "moe.cu", "gdn.cu", "step.cu", "ops.cu"):
        text = (csrc / name).read_text()
        for entry in re.finditer(r'extern "C" int qd_\w+\([^)]*\bint pdl\b[^)]*\) \{(.*?)\n\}', text, flags=re.S):
            assert re.search(r"pdl != 0|launch_mode\(pdl\)", entry.group(1)) and not re.search(r"[ (]pdl[,)] *(?!!)", entry.group(1).replace("launch_mode(pdl)", "")), name


def test_scratch_of_a_captured_step_outlives_a_larger_batch(monkeypatch):
    """A graph captured for a state holds the addresses of the attention's scratch and counters; a larger state's step replaces both, and
    the old ones must not go back to the allocator."""
    import weakref
    from types import SimpleNamespace

    from quickdraw_b200 import batch
    monkeypatch.setattr(batch, "lib", lambda: SimpleNamespace(qd_attn_scratch_floats=lambda *sizes: 8))
    decoder = batch.BatchDecode.__new__(batch.BatchDecode)
    decoder.ckpt = SimpleNamespace(config=SimpleNamespace(num_attention_heads=4, num_key_value_heads=2, head_dim=256))
    decoder.device, decoder._scratch, decoder._retired = "cpu", None, []
    small = decoder._attn_scratch(2)
    assert decoder._attn_scratch(1) == small and not decoder._retired
    alive = [weakref.ref(t) for t in small]
    addresses = [t.data_ptr() for t in small]
    del small
    large = decoder._attn_scratch(32)
    assert [r() is not None and r().data_ptr() for r in alive] == addresses
    assert [t.numel() for t in large] == [256, 64]


def test_splits_of_the_decode_attention_follow_the_form_that_is_taken():
    from quickdraw_b200.kernels import _attn_splits
    assert [_attn_splits(256, r, 4096) for r in (0, 64, 256, 32, 96)] == [74, 74, 74, 32, 32]
    assert _attn_splits(128, 64, 4096) == 32 and _attn_splits(256, 64, 4096 | 4104) == 32


@pytest.mark.parametrize("rows,before,ids", [([], 0, [1, 2]), ([1, 2, 3], 0, [1, 2]), ([1, 2, 3], 1, [2, 3, 4]), ([1, 2, 3, 4], 1, [2, 9, 4]),
                                             ([1, 2, 3], 0, [7]), ([1, 2], 2, [3]), ([1, 2, 3], 1, [])])
def test_cache_rows_follow_the_tokens_one_by_one(rows, before, ids):
    """What a run of tokens does to the record of the cache's rows is what its tokens do one after the other."""
    from types import SimpleNamespace
    from quickdraw_b200.engine import Engine
    want, history = list(rows), list(rows[:before])
    for token in ids:
        at = len(history)
        if not (at < len(want) and want[at] == token):
            del want[at:]
            want.append(token)
        history.append(token)
    engine = SimpleNamespace(history=list(rows[:before]), _kv_tokens=list(rows))
    Engine._note(engine, ids)
    assert engine._kv_tokens == want and engine.history == history
