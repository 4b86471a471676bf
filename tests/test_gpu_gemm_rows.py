"""The grouped GEMM's converters (csrc/dequant_f16.cuh) at the row lengths where they take different loads: rows whose super-blocks lie the
same distance from a 16-byte boundary in every row and rows that differ in it, by words and by half words, odd numbers of super-blocks; and
block scales of either sign, zero and below the smallest normal fp16 number."""
import numpy as np
import pytest

from helpers import REL_TO_NORM, TYPES, rel_to_norm, to_dev
from zeromoe_b200 import synth

pytestmark = pytest.mark.gpu

SCALES_AT = {synth.Q2_K: (80, 82), synth.Q3_K: (108,), synth.Q4_K: (0, 2), synth.IQ2_XXS: (0,)}


def _odd_scales(w, qtype, rng):
    """the tensor with some super-scales negated, zero or subnormal"""
    w = w.copy()
    blocks = w.reshape(-1, synth.BLOCK_BYTES[qtype])
    for at in SCALES_AT[qtype]:
        d = blocks[:, at:at + 2].copy().view(np.float16)[:, 0]
        kind = rng.integers(0, 8, d.shape)
        d = np.where(kind == 0, -d, d)
        d = np.where(kind == 1, np.float16(0), d)
        d = np.where(kind == 2, np.float16(3.1e-6), d).astype(np.float16)
        blocks[:, at:at + 2] = d.reshape(-1, 1).view(np.uint8)
    return w


@pytest.mark.parametrize("qtype", TYPES)
@pytest.mark.parametrize("D,F", [(1280, 768), (768, 1280), (2816, 256), (1536, 2048)])
def test_rows_of_every_alignment(zlib, dev, qtype, D, F):
    """Against the decode kernels, whose integer sums the oracle pins.  The two differ by the rounding of a weight (at most two roundings
    to 11 bits where a min is subtracted) and of an activation to fp16: 2^-11 each at most, in sums of independent signs, and the same
    rounding moves an 8-bit code of the activation now and then: the bounds of the other tests of this kernel."""
    import torch
    counts = [3, 48, 90, 17]
    E, T = len(counts), sum(counts)
    rng = synth.rng_for(83, D, F, qtype)
    ids = rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int32).reshape(T, 1)
    w = [_odd_scales(synth.expert_weights(qtype, E, o, i, rng), qtype, rng) for o, i in ((F, D), (F, D), (D, F))]
    x = synth.activations(T, D, rng)
    ctx = zlib.Context(T, D, F, E, 1)
    layer = zlib.Layer(ctx, D, F, E, 1, (qtype,) * 3, *[to_dev(a, dev) for a in w])
    outs = {}
    xd, idd, wtd = to_dev(x, dev), to_dev(ids, dev), to_dev(np.ones((T, 1), np.float32), dev)
    for path in (1, 2):
        ctx.set_path(path)
        layer.set_routes(xd, idd, wtd)
        out = torch.full((T, D), float("nan"), device=dev)
        layer.expert_ffn(out)
        torch.cuda.synchronize()
        ctx.check()
        outs[path] = (ctx.act(T, F).copy(), out.cpu().numpy())
    # the grouped GEMM ran, and not the decode kernels a second time: its weights and activations are fp16
    assert not np.array_equal(outs[2][0], outs[1][0])
    for got, ref in zip(outs[2], outs[1]):
        got, ref = got.reshape(T, -1), ref.reshape(T, -1)
        assert np.isfinite(got).all()
        assert rel_to_norm(got, ref) < REL_TO_NORM
        assert (np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)).max() < 2e-2
