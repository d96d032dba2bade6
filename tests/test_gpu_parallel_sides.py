"""The two sides of a parallel mixer on streams of their own against one after the other."""
import numpy as np
import pytest
import torch

from singe_b200 import models
from singe_b200.parallel_mixer import ChunkedAttention, GatedDelta, ParallelMixer
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


# few sequences, and enough for the decode attention that takes every SM's shared memory (with 16-bit activations)
@pytest.mark.parametrize("sequences,filling,dtype", [(2, False, "bfloat16"), (24, True, "bfloat16"), (24, False, "float32")])
@pytest.mark.parametrize("captured", [False, True])
def test_sides_beside_each_other(tmp_path, monkeypatch, sequences, filling, dtype, captured):
    directory = util.write_snapshot(tmp_path, CONFIG, util.make_weights(CONFIG, seed=3))
    if not captured:        # (left alone, only captured steps fork)
        monkeypatch.setattr(ParallelMixer, "beside", lambda self, step: step.longest <= 1)

    def steps():
        decoder = models.load_decoder(directory, sequences, 2048, dtype)
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


def test_a_side_is_waited_for_when_the_other_one_is_refused(tmp_path, monkeypatch):
    decoder = models.load_decoder(util.write_snapshot(tmp_path, CONFIG, util.make_weights(CONFIG, seed=3)), 2, 2048, "bfloat16")
    decoder.fill_context(100, seed=5)

    def busy(self, stream, *_):
        with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
            torch.cuda._sleep(400_000_000)     # a fifth of a second
        return lambda: None

    def refused(self, stream, *_):
        raise RuntimeError("refused")

    monkeypatch.setattr(ParallelMixer, "beside", lambda self, step: True)
    monkeypatch.setattr(GatedDelta, "prepare", busy)
    monkeypatch.setattr(ChunkedAttention, "prepare", refused)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="refused"):
        decoder.step(np.asarray([1, 2]))
    assert not torch.cuda.current_stream().query()
    torch.cuda.synchronize()


@pytest.mark.parametrize("captured", [False, True])
def test_only_captured_steps_fork(tmp_path, monkeypatch, captured):
    decoder = models.load_decoder(util.write_snapshot(tmp_path, CONFIG, util.make_weights(CONFIG, seed=3)), 2, 2048, "bfloat16")
    decoder.fill_context(100, seed=5)
    streams = []
    prepare = GatedDelta.prepare
    monkeypatch.setattr(GatedDelta, "prepare", lambda self, stream, *rest: (streams.append(stream), prepare(self, stream, *rest))[1])
    if captured:
        decoder.capture()       # a warm-up ahead of the capture, then the capture
    else:
        decoder.step(np.asarray([1, 2]))
    torch.cuda.synchronize()
    layers = len(decoder.layers)
    own = {int(layer.mixer.ops._side[0].cuda_stream) for layer in decoder.layers if layer.mixer.ops._side}
    assert len(streams) == (2 * layers if captured else layers) and len(own) == (1 if captured else 0)
    assert [stream in own for stream in streams] == [False] * layers + [True] * layers * captured
