"""All layers by one native call against the parts one by one: the same kernels, so the same bits, for every kind of step."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,heads,kv_heads,dim,inter,layers,window,page", [
    (64, 4, 2, 16, 72, 1, None, 8), (256, 8, 2, 64, 640, 3, None, 16), (1024, 16, 8, 128, 3072, 2, 40, 16), (2056, 3, 3, 112, 520, 2, None, 32)])
def test_every_kind_of_step_gives_the_same_bits(hidden, heads, kv_heads, dim, inter, layers, window, page, monkeypatch):
    from xinfer_b200 import kernels
    from xinfer_b200.engine.runner import ModelRunner, StepInput
    from xinfer_b200.models import dense_layers
    cfg = dict(architectures=["Qwen3ForCausalLM"], vocab_size=300, hidden_size=hidden, intermediate_size=inter, num_hidden_layers=layers,
               num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=dim, rms_norm_eps=1e-6, rope_theta=10000.0,
               max_position_embeddings=2048, tie_word_embeddings=False, sliding_window=window)
    rng = np.random.default_rng(5)
    ids = lambda n: rng.integers(0, 300, size=n, dtype=np.int32)
    # portions of the step's requests, some of which go on from the step before
    script = [[(0, 1), (1, 33), (2, 300)], [(0, 5), (1, 1), (2, 1)], [(0, 1), (1, 1), (2, 1)], [(0, 1), (1, 1), (2, 1)], [(3, 32)], [(4, 4), (0, 2)]]
    tokens = [[ids(n) for _, n in step] for step in script]

    def run(native):
        monkeypatch.setattr(dense_layers, "ENABLED", native)
        r = ModelRunner.random(cfg, 7, dtype="bf16", block_size=page, num_blocks=64, max_num_seqs=5, max_model_len=512)
        slots = [r.open_request() for _ in range(5)]
        before, out = kernels.launch_counts(), []
        for i, (step, toks) in enumerate(zip(script, tokens)):
            out.append(r.step([StepInput(slots[b], t, range(len(t))) for (b, n), t in zip(step, toks)], allow_graph=i == 3).clone())
        r.check_errors()
        return torch.cat(out), {k: n - before.get(k, 0) for k, n in kernels.launch_counts().items() if n > before.get(k, 0)}

    a, count_a = run(True)
    b, count_b = run(False)
    count_a.pop("rope_table", None)         # (kept from the first run)
    assert torch.equal(a, b) and count_a == count_b


def test_other_stacks_keep_to_the_parts():
    from xinfer_b200.engine.runner import ModelRunner
    cfg = dict(architectures=["Qwen3ForCausalLM"], vocab_size=300, hidden_size=64, intermediate_size=64, num_hidden_layers=1, num_attention_heads=2,
               num_key_value_heads=1, head_dim=160, rms_norm_eps=1e-6, rope_theta=10000.0, max_position_embeddings=64, tie_word_embeddings=True)
    opts = dict(block_size=16, num_blocks=8, max_num_seqs=1, max_model_len=64)
    assert ModelRunner.random(cfg, 1, dtype="bf16", **opts).model.dense is None          # heads of more than 128 values
    assert ModelRunner.random(dict(cfg, head_dim=64), 1, dtype="f32", **opts).model.dense is None
    assert ModelRunner.random(dict(cfg, head_dim=64), 1, dtype="bf16", **opts).model.dense is not None


CFG = dict(architectures=["Qwen3ForCausalLM"], vocab_size=300, hidden_size=256, intermediate_size=640, num_hidden_layers=3, num_attention_heads=8,
           num_key_value_heads=2, head_dim=64, rms_norm_eps=1e-6, rope_theta=10000.0, max_position_embeddings=2048, tie_word_embeddings=False)


def steps(monkeypatch, native=True):
    """Logits of a prompt step, a mixed and a decode step."""
    from xinfer_b200.engine.runner import ModelRunner, StepInput
    from xinfer_b200.models import dense_layers
    monkeypatch.setattr(dense_layers, "ENABLED", native)
    r = ModelRunner.random(CFG, 7, dtype="bf16", block_size=16, num_blocks=64, max_num_seqs=3, max_model_len=512)
    slots = [r.open_request() for _ in range(3)]
    rng, out = np.random.default_rng(5), []
    for step in ([(0, 70), (1, 2)], [(2, 100), (0, 1), (1, 1)], [(0, 1), (1, 1), (2, 1)]):
        toks = [rng.integers(0, 300, size=n, dtype=np.int32) for _, n in step]
        out.append(r.step([StepInput(slots[b], t, range(len(t))) for (b, _), t in zip(step, toks)], allow_graph=False).clone())
    r.check_errors()
    return torch.cat(out)


class Library:
    """The native library with another ``xb_dense_layers``."""

    def __init__(self, lib, call):
        self._lib, self._call = lib, call

    def __getattr__(self, name):
        return self._call if name == "xb_dense_layers" else getattr(self._lib, name)


@pytest.mark.parametrize("switch", ["reduced precision", "library", "tunable"])
def test_torchs_switches_send_products_through_torch(switch, monkeypatch):
    from xinfer_b200 import kernels
    called = []
    whole = kernels.dense_layers
    monkeypatch.setattr(kernels, "dense_layers", lambda *a: (called.append(1), whole(*a)))
    steps(monkeypatch)
    assert len(called) == 3
    called.clear()
    blas = torch.backends.cuda.preferred_blas_library()
    try:
        if switch == "reduced precision":
            torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
        elif switch == "library":
            torch.backends.cuda.preferred_blas_library("cublaslt")
        else:
            monkeypatch.setattr(torch.cuda.tunable, "is_enabled", lambda: True)
        steps(monkeypatch)
    finally:
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = True
        torch.backends.cuda.preferred_blas_library(blas)
    assert not called


def test_without_torchs_library_the_parts_run(monkeypatch):
    import ctypes
    from xinfer_b200.engine.runner import ModelRunner

    def none(name, *a, **k):
        raise OSError(name)
    opts = dict(block_size=16, num_blocks=8, max_num_seqs=1, max_model_len=64)
    with monkeypatch.context() as m:
        m.setattr(ctypes, "CDLL", none)
        r = ModelRunner.random(CFG, 1, dtype="bf16", **opts)
        assert r.model.dense is None


@pytest.mark.parametrize("layer", [0, 2])
def test_an_attention_kernel_that_does_not_take_the_step(layer, monkeypatch):
    """Layer ``layer``'s attention is refused (and what its kernels have written is spoilt): another kernel attends and the call goes on."""
    import ctypes
    from xinfer_b200 import kernels, native
    from xinfer_b200.parts import attention_backend
    expect = steps(monkeypatch, native=False)
    real, types = native.kernels_lib(), kernels.dense_types()
    refused, attend = [], attention_backend.attend

    def refuse(step, layers, begin, end, done, stream):
        if begin > 2 * layer or end <= 2 * layer:
            return real.xb_dense_layers(step, layers, begin, end, done, stream)
        rc = real.xb_dense_layers(step, layers, begin, 2 * layer + 1, done, stream)
        report = ctypes.cast(done, ctypes.POINTER(types[2])).contents
        report.half, report.launch = 2 * layer, 4
        refused.append(report.half)
        return rc or kernels.ERR_NOT_SUPPORTED

    def attended(out, *a, **k):
        out.fill_(float("nan"))
        attend(out, *a, **k)
    monkeypatch.setattr(kernels, "kernels_lib", lambda: Library(real, refuse))
    monkeypatch.setattr(attention_backend, "attend", attended)
    got = steps(monkeypatch)
    assert refused == [2 * layer] * 3 and torch.equal(got, expect)


def test_the_error_names_what_failed(monkeypatch):
    import ctypes
    from xinfer_b200 import kernels, native
    real, types = native.kernels_lib(), kernels.dense_types()

    def fail(step, layers, begin, end, done, stream):
        report = ctypes.cast(done, ctypes.POINTER(types[2])).contents
        report.half, report.launch, report.blas_status = 3, 2, 13
        return 999
    monkeypatch.setattr(kernels, "kernels_lib", lambda: Library(real, fail))
    with pytest.raises(kernels.KernelError, match=r"library product of layer 1 \(cuBLAS status 13\): CUDA error 999"):
        steps(monkeypatch)


def test_the_mirrors_members_have_the_librarys_names():
    from xinfer_b200 import kernels
    step, layer, done = kernels.dense_types()
    assert [n for n, _ in step._fields_][:3] == ["x", "h", "qkv"] and [n for n, _ in step._fields_][-2:] == ["p0", "p1"]
    assert [n for n, _ in layer._fields_] == "w_qkv w_o w_gate_up w_down norm1 norm2 q_norm k_norm k_pages v_pages".split()
    assert [n for n, _ in done._fields_][3:] == "norms skinny library ropes prefill decode gates".split()
