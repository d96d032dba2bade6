"""The two sides of a parallel mixer on streams of their own against one after the other."""
import numpy as np
import pytest
import torch

from singe_b200 import models
from singe_b200.parallel_mixer import ParallelMixer
from tests import vatolorn_util as util

pytestmark = pytest.mark.gpu

CONFIG = util.model(256, 300, 4, 0.7, 1e-5,
                    util.layer(util.left(8, 4, 64, 64, 4096, 4, util.rot(64, 10000.0, (8.0, 128, 32.0, 1.0)), 0.125),
                               util.right(8, 8, 64, 128, 4), 512),
                    util.layer(util.left(16, 8, 128, 128, 1024, 3, util.rot(64, 10000.0, (8.0, 128, 32.0, 1.0)), 0.1),
                               util.right(4, 2, 64, 64, 2), 320))


def one_after_the_other(self, stream, step, normed, cache, delta, status, scratch=None):
    projected = self.ops.rows(normed.shape[0], self.project.shape[0])
    self.ops.linear(stream, projected, normed, self.project)
    width = normed.shape[1]
    self.left.prepare(stream, step, projected[:, :self.split], cache[:3], delta[:, :width], status, scratch)()
    self.right.prepare(stream, step, projected[:, self.split:], cache[3:], delta[:, delta.shape[1] - width:], status)()


# few sequences, and enough for the decode attention that takes every SM's shared memory
@pytest.mark.parametrize("sequences,filling", [(2, False), (24, True)])
@pytest.mark.parametrize("captured", [False, True])
def test_sides_beside_each_other(tmp_path, monkeypatch, sequences, filling, captured):
    directory = util.write_snapshot(tmp_path, CONFIG, util.make_weights(CONFIG, seed=3))

    def steps():
        decoder = models.load_decoder(directory, sequences, 2048, "bfloat16")
        bound = decoder.stride * 16
        assert {layer.mixer.left.fills_machine(sequences, bound) for layer in decoder.layers} == {filling}
        decoder.fill_context(700, seed=5)
        if captured:
            decoder.capture()
        out = []
        for i in range(4):
            tokens = np.random.default_rng(i).integers(0, CONFIG["vocab"], size=sequences)
            decoder.step(tokens)
            out.append(decoder.logits.clone())
        torch.cuda.synchronize()
        assert int(decoder.status.item()) == 0
        return out, [part.clone() for cache in decoder.caches for part in cache]

    beside = steps()
    monkeypatch.setattr(ParallelMixer, "run", one_after_the_other)
    for mine, other in zip(beside, steps()):
        assert all(torch.equal(a, b) for a, b in zip(mine, other))
