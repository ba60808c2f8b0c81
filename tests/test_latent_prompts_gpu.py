"""Attention over latents for prompts from position 0: keys and values of every head made from the latents, against 64 bits, beside the way through the latent, and in graphs."""
from __future__ import annotations

import pytest
import torch

from hyperion_b200.api import Engine, resolve_dtype
from hyperion_b200.engine.batch import StepEntry
from hyperion_b200.models import DecoderModel, architecture_of
from hyperion_b200.parts import attention_latent

pytestmark = pytest.mark.gpu
WIDTH, RANK, QRANK, VOCAB = 256, 128, 192, 300


def _engine(heads, dim, rot, vdim, page_size, room, rows):
    mixer = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": RANK, "q_rank": QRANK, "scale": (dim + rot) ** -0.5, "rot": {"dims": rot, "base": 1e4}}
    document = {"architecture": "Kudazen", "vocab": VOCAB, "width": WIDTH, "norm": {"eps": 1e-6, "groups": 1},
                "layers": [{"type": "latent_attention", "mlp": {"kind": "dense", "ff": 128, "limit": 7.0}, "mixer": mixer}]}
    architecture = architecture_of(document)
    config = architecture.read_config(document)
    model = DecoderModel(architecture.build_spec(config), resolve_dtype("bfloat16"), torch.device("cuda:0"))
    g = torch.Generator("cuda").manual_seed(heads)
    tensors = {}
    for name, wanted in model.expected_tensors().items():
        std = 1.0 if name == "embed" or name.endswith("sink") else 0.1 if "norm" in name else 0.7 if ".uq" in name else wanted.shape[-1] ** -0.5
        tensors[name] = (torch.randn(wanted.shape, device="cuda", generator=g) * std + (1.0 if "norm" in name else 0.0)).to(torch.bfloat16)
    model.load(tensors)
    return Engine(model, config, page_size=page_size, max_tokens=room, max_requests=rows), model, {n: t.double() for n, t in tensors.items()}


def _exact(w, heads, dim, rot, vdim, ids):
    """Logits at every place in 64 bits."""
    def unit(x, name):
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * w[name]

    def turned(x):
        T = x.shape[0]
        angle = torch.arange(T, device="cuda", dtype=torch.float64)[:, None, None] * 1e4 ** (-2.0 * torch.arange(rot // 2, device="cuda", dtype=torch.float64) / rot)
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin()], -1).flatten(-2)

    x = w["embed"][torch.tensor(ids, device="cuda")]
    h = unit(x, "l0.norm1")
    q = (unit(h @ w["l0.mix.dq"].T, "l0.mix.dq.norm") @ w["l0.mix.uq"].T).view(len(ids), heads, dim + rot)
    down = h @ w["l0.mix.dkv"].T
    latent = unit(down[:, :RANK], "l0.mix.dkv.norm")
    k = torch.cat([(latent @ w["l0.mix.uk"].T).view(-1, heads, dim), turned(down[:, None, RANK:]).expand(-1, heads, -1)], -1)
    q = torch.cat([q[..., :dim], turned(q[..., dim:])], -1)
    s = torch.einsum("ihd,jhd->hij", q, k) * (dim + rot) ** -0.5
    s = s.masked_fill(torch.ones(len(ids), len(ids), dtype=torch.bool, device="cuda").triu(1), -torch.inf)
    z = w["l0.mix.sink"][:, None, None]
    top = torch.maximum(s.amax(-1, keepdim=True), z)
    p = torch.exp(s - top)
    p = p / (p.sum(-1, keepdim=True) + torch.exp(z - top))
    o = torch.einsum("hij,jhe->ihe", p, (latent @ w["l0.mix.uv"].T).view(-1, heads, vdim)).flatten(1)
    g = (h @ w["l0.mlp.gate"].T).clamp(max=7.0)
    u = (h @ w["l0.mlp.up"].T).clamp(-7.0, 7.0)
    return unit(x + o @ w["l0.mix.o"].T + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w["l0.mlp.down"].T, "final.norm") @ w["embed"].T


# prompts that end inside a page and a tile, at their ends, of few tokens beside long ones; the shared part of a key wide and narrow
@pytest.mark.parametrize("heads,dim,rot,vdim", [(4, 128, 64, 128), (3, 96, 96, 128), (1, 176, 16, 128)])
@pytest.mark.parametrize("lengths,page_size", [((512,), 16), ((900, 64, 5), 8), ((300, 301), 64), ((128, 1, 384), 16)])
def test_prompts(heads, dim, rot, vdim, lengths, page_size, monkeypatch):
    engine, model, w = _engine(heads, dim, rot, vdim, page_size, 4 * sum(lengths) + 512, 8)
    assert model.layers[0].mixer.expands_fresh_prompts
    g = torch.Generator().manual_seed(heads)
    prompts = [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in lengths]
    taken = []
    real = attention_latent.LatentAttention._attend_expanded
    monkeypatch.setattr(attention_latent.LatentAttention, "_attend_expanded", lambda self, *a: taken.append(1) or real(self, *a))

    def run(whole=True):
        want = [[0, len(p) // 2, len(p) - 1] for p in prompts]
        if whole:
            out = engine.step([StepEntry(i, p, at) for i, (p, at) in enumerate(zip(prompts, want))]).clone()
        else:  # the first token, then the rest: no step of prompts from position 0
            first = engine.step([StepEntry(i, p[:1], [0]) for i, p in enumerate(prompts)]).clone()
            rest = engine.step([StepEntry(i, p[1:], [a - 1 for a in at[1:]]) for i, (p, at) in enumerate(zip(prompts, want))]).clone().view(len(prompts), 2, -1)
            out = torch.cat([first[:, None], rest], 1).flatten(0, 1)
        engine.runner.check_device_status()
        for i in range(len(prompts)):
            engine.finish(i)
        return out

    runs = [run() for _ in range(4)]  # direct, direct, captured, replayed
    if min(lengths) <= 4:  # a row that goes token by token: the whole step keeps to the latent
        assert not taken
        return
    assert len(taken) == 3 and all(torch.equal(runs[0], r) for r in runs[1:])
    through_latent = run(whole=False)
    assert len(taken) == 3
    exact = torch.cat([_exact(w, heads, dim, rot, vdim, p)[[0, len(p) // 2, len(p) - 1]] for p in prompts])
    far, as_far = ((o.double() - exact).norm() / exact.norm() for o in (runs[0], through_latent))
    assert far <= 0.02 and far <= 1.3 * as_far + 1e-4, (far, as_far)  # both round what enters a product to bfloat16, at other places


def test_a_graph_of_prompts_is_not_replayed_for_their_continuation():
    """Steps of the same shape, from position 0 and behind earlier tokens, in turn."""
    engine, _, w = _engine(4, 128, 64, 128, 16, 16384, 4)
    g = torch.Generator().manual_seed(1)
    ids = torch.randint(0, VOCAB, (1200,), generator=g).tolist()
    exact = _exact(w, 4, 128, 64, 128, ids)
    for _ in range(5):
        first = engine.step([StepEntry("a", ids[:600], [599])]).clone()
        second = engine.step([StepEntry("a", ids[600:], [599])]).clone()
        engine.finish("a")
        for got, at in ((first, 599), (second, 1199)):
            assert (got[0].double() - exact[at]).norm() <= 0.02 * exact[at].norm()
