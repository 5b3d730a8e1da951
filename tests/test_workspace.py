"""Scratch buffers (CPU): those whose size follows the context."""
import pytest
import torch

from xinfer_b200.parts.base import Workspace


def test_context_scratch_grows_in_few_steps_and_not_beyond_its_most():
    ws, sizes = Workspace("cpu"), []
    for n in range(100, 5001, 100):
        assert ws.reserve("a", n, torch.float32, 4100)
        assert ws.get("a", (n // 10, 10), torch.float32).shape == (n // 10, 10)
        sizes.append(ws.bytes() // 4)
    assert sizes[0] == 128 and sizes[sizes.index(4100) - 1] == 4096 and sizes[-1] == 5000
    assert len({s for s in sizes if s <= 4100}) == 7            # 128, 256, ... 4,096, 4,100


def test_a_device_without_room_says_so_once_and_again_after_a_reset(monkeypatch):
    ws, asked = Workspace("cpu"), []
    empty = torch.empty

    def full(n, **kw):
        asked.append(n)
        if n > 300:
            raise torch.OutOfMemoryError("no room")
        return empty(n, **kw)
    monkeypatch.setattr(torch, "empty", full)
    assert ws.reserve("a", 200, torch.float32, 1 << 20) and asked == [256]
    assert ws.reserve("a", 290, torch.float32, 1 << 20) and asked == [256, 512, 290]      # just what is needed, where slack is too much
    assert not ws.reserve("a", 400, torch.float32, 1 << 20) and asked[3:] == [512, 400]
    assert not ws.reserve("a", 500, torch.float32, 1 << 20) and len(asked) == 5           # not tried again
    assert ws.reserve("a", 100, torch.float32, 1 << 20)
    ws.clear()
    assert not ws.reserve("a", 400, torch.float32, 1 << 20) and len(asked) == 8


def test_a_buffer_that_a_graph_uses_does_not_move():
    ws = Workspace("cpu")
    assert ws.reserve("a", 100, torch.float32, 1000)
    ws.frozen = True
    assert ws.reserve("a", 128, torch.float32, 1000)
    with pytest.raises(RuntimeError, match="'a'"):
        ws.reserve("a", 129, torch.float32, 1000)


def test_a_model_names_the_scratch_that_follows_the_context():
    from xinfer_b200.config import config_from_dict
    from xinfer_b200.models.decoder import DecoderModel
    from xinfer_b200.parts import latent_attention, talking_attention
    rot = dict(dims=32, base=1000.0)
    latent = dict(type="latent_attention", mlp=dict(kind="dense", ff=128, limit=7.0),
                  mixer=dict(heads=2, dim=64, rot_dim=32, vdim=64, q_rank=96, kv_rank=64, scale=0.1, rot=rot))
    napuzen = dict(architecture="Napuzen", vocab=300, width=128, norm=dict(eps=1e-6), canon=dict(taps=4), logit_scale=0.8, layers=[latent, latent])
    left = dict(heads=8, kv_heads=4, dim=64, vdim=64, scale=0.125, rot=dict(dims=64, base=1000.0))
    talk = dict(type="parallel", mixer=dict(left=left, left_scale=0.5, right=dict(width=64), right_scale=1.0), mlp=dict(kind="dense", ff=128))
    tidarax = dict(architecture="Tidarax", vocab=300, width=128, norm=dict(eps=1e-6), layers=[talk, talk])
    for cfg, want in ((napuzen, latent_attention.ROWS_MAX_BYTES * (1 + 96 / 256)), (tidarax, talking_attention.SCORES_BYTES)):
        entry, parsed = config_from_dict(cfg)
        for dtype, most in ((torch.bfloat16, want), (torch.float32, 0)):
            assert DecoderModel(entry.plan_of(parsed), dtype, "cpu").context_scratch_bytes() == most     # once, though two layers use it
