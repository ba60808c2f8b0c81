"""Attention over latents inside a wrapper: graphs of prompts from position 0 and of their continuations stay apart as they do without one."""
from __future__ import annotations

import dataclasses

import pytest
import torch

import test_latent_prompts_gpu as plain
from hyperion_b200.engine.batch import StepEntry
from hyperion_b200.models import DecoderModel
from hyperion_b200.parts.spec import PartSpec

pytestmark = pytest.mark.gpu


def test_a_graph_of_prompts_is_not_replayed_for_their_continuation(monkeypatch):
    def wrapped(spec, *rest):
        layer = spec.layers[0]
        mixer = PartSpec("input_convolution", "", {"hidden_size": plain.WIDTH, "taps": 1, "weight_name": "conv0", "inner": layer.mixer})
        return DecoderModel(dataclasses.replace(spec, layers=(dataclasses.replace(layer, mixer=mixer),)), *rest)

    monkeypatch.setattr(plain, "DecoderModel", wrapped)
    engine, model, w = plain._engine(4, 128, 64, 128, 16, 16384, 4)
    model.layers[0].mixer.weight.zero_()  # the inner mixer reads its rows as they are
    assert model.layers[0].mixer.inner.expands_fresh_prompts
    ids = torch.randint(0, plain.VOCAB, (1200,), generator=torch.Generator().manual_seed(1)).tolist()
    exact = plain._exact(w, 4, 128, 64, 128, ids)
    for _ in range(5):
        first = engine.step([StepEntry("a", ids[:600], [599])]).clone()
        second = engine.step([StepEntry("a", ids[600:], [599])]).clone()
        engine.finish("a")
        for got, at in ((first, 599), (second, 1199)):
            assert (got[0].double() - exact[at]).norm() <= 0.02 * exact[at].norm()
