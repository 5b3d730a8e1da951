"""Rows in vectors against 64 bits: widths around a thread's vectors, every combination of the row's operands, gathered rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dim", [4, 252, 256, 516, 1024, 4096, 4100, 8192])
@pytest.mark.parametrize("branch,norm,gain,scale,weight,rows", [
    (None, False, False, 1.0, True, False), (torch.float32, True, True, 0.5, True, False), (torch.bfloat16, True, False, 1.0, False, False),
    (torch.bfloat16, False, True, 2.0, True, True), (torch.float32, False, False, 1.0, True, True)])
def test_rows_in_vectors(dim, branch, norm, gain, scale, weight, rows):
    from xinfer_b200 import kernels as k
    g = torch.Generator().manual_seed(dim)
    n = 5
    x = torch.randn(n, dim, generator=g)
    br = torch.randn(n, dim, generator=g).to(branch) if branch else None
    w, bw, gn = (1 + 0.1 * torch.randn(dim, generator=g) for _ in range(3))
    idx = [4, 0, 2] if rows else list(range(n))
    to = lambda t: None if t is None else t.to(DEV)
    out = torch.empty(len(idx), dim, dtype=torch.bfloat16, device=DEV)
    total = torch.empty(len(idx), dim, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    k.rms_chain(out, to(x), to(w) if weight else None, 1e-5, err, branch=to(br), branch_weight=to(bw) if norm else None, branch_eps=1e-6,
                branch_offset=0.25, gain=to(gn) if gain else None, branch_scale=scale, sum_out=total,
                rows=torch.tensor(idx, dtype=torch.int32, device=DEV) if rows else None, weight_offset=0.5)
    s = x.double()
    if br is not None:
        b = br.double()
        if norm:
            b = b * torch.rsqrt((b * b).mean(1, keepdim=True) + 1e-6) * (0.25 + bw.double())
        s = s + scale * (gn.double() if gain else 1.0) * b
    y = s * torch.rsqrt((s * s).mean(1, keepdim=True) + 1e-5) * (0.5 + w.double()) if weight else s
    assert int(err) == 0
    assert (total.double().cpu() - s[idx]).abs().max() <= 2e-6 * (1 + s.abs().max())      # a few float32 roundings
    assert (out.double().cpu() - y[idx]).abs().max() <= 2.0 ** -8 * y.abs().max()         # one to bfloat16


@pytest.mark.parametrize("rows,width", [(65, 4), (66, 1020), (600, 1028), (2000, 3072)])
@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
def test_gate_with_biases_over_many_rows_gives_the_bits_of_few(rows, width, activation):
    from xinfer_b200 import kernels as k
    g = torch.Generator().manual_seed(width)
    gu, bias = torch.randn(rows, 2 * width, generator=g).to(DEV), torch.randn(2 * width, generator=g).to(DEV)
    out, few = (torch.zeros(rows, width, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    k.swiglu_bias(out, gu, bias, activation)
    for a in range(0, rows, 64):
        k.swiglu_bias(few[a:a + 64], gu[a:a + 64], bias, activation)
    assert torch.equal(out, few)


@pytest.mark.parametrize("T,parts,part", [(3, 2, 4), (9, 3, 128), (5, 2, 132), (2, 3, 512), (2, 2, 516), (3, 2, 1024), (2, 1, 1028), (2, 1, 4096), (2, 1, 4100)])
@pytest.mark.parametrize("after,silu,div", [(False, False, False), (True, False, True), (True, True, False)])
def test_gated_parts_in_vectors(T, parts, part, after, silu, div):
    from xinfer_b200 import kernels as k
    g = torch.Generator().manual_seed(part)
    W, eps = parts * part, 1e-6
    y, gate, w = torch.randn(T, W, generator=g), torch.randn(T, W + 8, generator=g), 1 + torch.rand(part, generator=g)
    d = torch.rand(T, parts, generator=g) + 0.5
    d[-1, 0] = 0.0
    out = torch.full((T, W + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    k.gated_head_norm(out[:, 4:4 + W], y.to(DEV), gate.to(DEV), 4, w.to(DEV), part, eps, after, silu, div=d.to(DEV) if div else None, out_scale=-2.0)
    v, z = y.double().view(T, parts, part), gate.double()[:, 4:4 + W].reshape(T, parts, part)
    if div:
        v = v / torch.where(d == 0, 1.0, d.double())[..., None]
    if not after:
        v = v * z * torch.sigmoid(z)
    v = v * (v.square().mean(-1, keepdim=True) + eps).rsqrt() * w.double() * -2.0
    if after:
        v = v * torch.sigmoid(z) * (z if silu else 1.0)
    got = out.double().cpu()
    assert (got[:, :4] == 7.0).all() and (got[:, 4 + W:] == 7.0).all()
    assert ((got[:, 4:4 + W] - v.reshape(T, W)).abs() <= 2.0 ** -8 * v.reshape(T, W).abs() + 1e-5).all()     # one rounding to bfloat16, float32 behind it


def same(a, b):
    """Numbers of the same bits, and no number at the same places."""
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a, nan=0.0), torch.nan_to_num(b, nan=0.0))


BAD = [float("inf"), float("-inf"), float("nan"), 3e38, 1e20]


@pytest.mark.parametrize("where", ["x", "branch"])
def test_rows_in_vectors_with_infinities_as_the_general_kernel_has_them(where):
    """Rows that start off a 16-byte boundary run on the general kernel; a row's bad number reaches that row alone."""
    from xinfer_b200 import kernels as k
    g = torch.Generator().manual_seed(1)
    n, dim = len(BAD) + 1, 1024
    x, br = torch.randn(n, dim, generator=g).to(DEV), torch.randn(n, dim, generator=g).to(DEV)
    for i, v in enumerate(BAD):
        (x if where == "x" else br)[i, 77 * (i + 1)] = v
    w = (1 + 0.1 * torch.randn(dim, generator=g)).to(DEV)
    off = torch.empty(n * dim + 1, device=DEV)[1:].view(n, dim)
    off.copy_(x)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    for norm in (None, w):
        a, b = (torch.empty(n, dim, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        k.rms_chain(a, x, w, 1e-5, err, branch=br, branch_weight=norm, branch_eps=1e-6)
        k.rms_chain(b, off, w, 1e-5, err, branch=br, branch_weight=norm, branch_eps=1e-6)
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.isnan(a[:3]).any(1).all() and torch.isfinite(a[3:]).all()
        fine = ~torch.isnan(a)
        assert ((a[fine].float() - b[fine].float()).abs() <= 2.0 ** -7 * b[fine].float().abs()).all()      # one rounding apart


@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
def test_gate_over_many_rows_with_infinities(activation):
    from xinfer_b200 import kernels as k
    g = torch.Generator().manual_seed(2)
    rows, width = 70, 64
    gu, bias = torch.randn(rows, 2 * width, generator=g).to(DEV), torch.zeros(2 * width, device=DEV)
    for i, v in enumerate(BAD):
        gu[i, 3], gu[10 + i, width + 5] = v, v
    out, few = (torch.zeros(rows, width, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    k.swiglu_bias(out, gu, bias, activation)
    k.swiglu_bias(few[:35], gu[:35], bias, activation)
    k.swiglu_bias(few[35:], gu[35:], bias, activation)
    assert same(out, few) and torch.isfinite(out[20:]).all()


@pytest.mark.parametrize("part", [64, 512, 1028])
@pytest.mark.parametrize("after", [False, True])
def test_gated_parts_with_infinities_as_the_general_kernel_has_them(part, after):
    """Gates whose columns start off a 16-byte boundary send the call to the general kernel."""
    from xinfer_b200 import kernels as k
    g = torch.Generator().manual_seed(3)
    T, W = len(BAD) + 1, 2 * part
    y, gate, w = torch.randn(T, W, generator=g).to(DEV), torch.randn(T, W + 8, generator=g).to(DEV), torch.ones(part, device=DEV)
    for i, v in enumerate(BAD):
        y[i, 5] = v
    out, general = (torch.empty(T, W, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    k.gated_head_norm(out, y, gate, 4, w, part, 1e-6, after)
    other = torch.empty_like(gate)
    other[:, 5:5 + W] = gate[:, 4:4 + W]
    k.gated_head_norm(general, y, other, 5, w, part, 1e-6, after)
    assert torch.equal(torch.isnan(out), torch.isnan(general)) and torch.isfinite(out[:, part:]).all() and torch.isfinite(out[-1]).all()
    fine = ~torch.isnan(out)
    assert ((out[fine].float() - general[fine].float()).abs() <= 2.0 ** -7 * general[fine].float().abs()).all()
