"""Kernels that start before their predecessor has ended read and write nothing before its end: chains of dependent launches,
at grids and portions on both sides of the rule, give the numbers of launches with a synchronisation between them."""
import numpy as np
import pytest
import torch

from xinfer_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 147, 148, 149, 600])
def test_a_chain_of_sums_is_exact(blocks):
    n = blocks * 256
    step = torch.randint(-3, 4, (n,), device="cuda:0").to(torch.bfloat16)
    a, b = torch.zeros(n, device="cuda:0"), torch.full((n,), float("nan"), device="cuda:0")
    for _ in range(50):
        kernels.add(b, a, step)
        kernels.add(a, b, step)
    assert torch.equal(a, 100 * step.float())            # whole numbers: exact in float32


@pytest.mark.parametrize("tokens", [1, 8, 9, 33])
def test_a_chain_of_scans_carries_its_state(tokens):
    H, P, N, B = 4, 32, 32, 3
    g = torch.Generator(device="cuda:0").manual_seed(tokens)
    T = tokens * B
    xbc, proj = torch.randn(T, H * P + 2 * N, generator=g, device="cuda:0"), torch.randn(T, H, generator=g, device="cuda:0")
    bias, a_log, skip = (torch.randn(H, generator=g, device="cuda:0") for _ in range(3))
    q_start = torch.arange(B + 1, dtype=torch.int32, device="cuda:0") * tokens
    slots = torch.tensor([2, 0, 1], dtype=torch.int32, device="cuda:0")

    def chain(wait):
        state = torch.zeros(B, H, N, P, device="cuda:0")
        out = [torch.empty(T, H * P, device="cuda:0") for _ in range(12)]
        for y in out:
            kernels.selective_scan(y, xbc, proj, 0, bias, a_log, skip, state, q_start, slots, B, H, P, N, 1)
            if wait:
                torch.cuda.synchronize()
        return torch.stack(out), state
    for got, want in zip(chain(False), chain(True)):
        assert torch.equal(got, want)


@pytest.mark.parametrize("d,dv", [(64, 64), (64, 128), (128, 64)])
def test_attention_with_room_beside_it_runs_in_front_of_a_product_of_few_tokens(d, dv):
    # Both allocate tensor memory, and at these sizes a processor has shared memory for a block of each.
    H, rank, T, start = 40, 64, 8, 700
    g = torch.Generator(device="cuda:0").manual_seed(d + dv)
    bf = lambda *s: torch.randn(*s, generator=g, device="cuda:0").bfloat16()
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device="cuda:0")
    host, ctas, n, _ = kernels.latent_prefill_work([T], [start], 4, None, H)
    work, q, kv, rows, w = host.to("cuda:0"), bf(T, H * d), bf(n, H * (d + dv)), bf(n, rank), bf(512, H * dv)
    q_start, start_pos, err = i32([0, T]), i32([start]), i32([0])

    def chain(wait):
        out, y = torch.zeros(T, H * dv, dtype=torch.bfloat16, device="cuda:0"), [torch.empty(T, 512, device="cuda:0") for _ in range(20)]
        for one in y:
            kernels.attn_rows_tc(out, q, H * d, kv, rows, work, ctas, q_start, start_pos, H, d, 0, dv, rank, None, d ** -0.5, None, err)
            if wait:
                torch.cuda.synchronize()
            assert kernels.gemm_skinny_tc(one, out, w, err)
        torch.cuda.synchronize()
        return torch.stack(y)
    assert torch.equal(chain(False), chain(True)) and int(err) == 0
