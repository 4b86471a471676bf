"""Layers with a clamped SwiGLU, in both forms of the clamp, through every kernel that has the activation in its epilogue."""
import numpy as np
import pytest

from helpers import REL_TO_NORM, rel_to_norm, to_dev
from zeromoe_b200 import synth

pytestmark = pytest.mark.gpu
D, F, E, K = 512, 512, 4, 2


def _layer(zlib, oracle, dev, qtype, T, fused, seed):
    """weights, routes, and a clamp that cuts into the values: the median magnitude of an unclamped result, or its root where the clamp is on gate and
    up, of which it is the product"""
    rng = synth.rng_for(seed, qtype, T)
    w = [synth.expert_weights(qtype, E, o, i, rng) for o, i in ((F, D), (F, D), (D, F))]
    x = synth.activations(T, D, rng)
    ids = np.stack([np.arange(T) % E, (np.arange(T) + 1) % E], axis=1).astype(np.int32)
    wts = np.full((T, K), 0.5, dtype=np.float32)
    free = oracle.moe_ffn(oracle.make_layer(D, F, E, K, (qtype,) * 3, *w), x, ids, wts, want_act=True)[1]
    clamp = float(np.median(np.abs(free)))
    if fused:
        clamp = clamp ** 0.5
    ref = oracle.moe_ffn(oracle.make_layer(D, F, E, K, (qtype,) * 3, *w, clamp=clamp, fused=fused), x, ids, wts, want_act=True)
    assert (ref[1] != free).mean() > 0.1
    return w, x, ids, wts, clamp, ref


@pytest.mark.parametrize("fused", [0, 1])
@pytest.mark.parametrize("path", [1, 2])
@pytest.mark.parametrize("qtype", [synth.Q2_K, synth.IQ2_XXS])
def test_clamped_layer_vs_oracle(zlib, oracle, dev, qtype, path, fused):
    """the decode kernels and the grouped GEMM, whose epilogue has a form of its own for a clamp; and a gate row that is not a number, which the clamp
    on the gate hides from the result but not from the counters"""
    import torch
    T = 48
    w, x, ids, wts, clamp, (ref, ref_act) = _layer(zlib, oracle, dev, qtype, T, fused, 88)
    ctx = zlib.Context(T, D, F, E, K)
    ctx.set_path(path)
    bad = w[0].copy()
    at = {synth.Q2_K: 80, synth.IQ2_XXS: 0}[qtype]
    bad[1, 5, at:at + 2] = (0x00, 0x7E)          # NaN in the first super-scale of expert 1's gate row 5
    xd, idd, wtd = to_dev(x, dev), to_dev(ids, dev), to_dev(wts, dev)
    for gate, nans in ((w[0], 0), (bad, T * K // E)):
        layer = zlib.Layer(ctx, D, F, E, K, (qtype,) * 3, to_dev(gate, dev), to_dev(w[1], dev), to_dev(w[2], dev), clamp=clamp, clamp_fused=fused)
        layer.set_routes(xd, idd, wtd)
        out = torch.empty((T, D), device=dev)
        layer.expert_ffn(out)
        torch.cuda.synchronize()
        ctx.check()
        assert ctx.bad_counts() == (nans, 0)
        if not nans:
            assert rel_to_norm(ctx.act(T * K, F).reshape(ref_act.shape), ref_act) < REL_TO_NORM
            assert rel_to_norm(out.cpu().numpy(), ref) < REL_TO_NORM


@pytest.mark.parametrize("fused", [0, 1])
def test_clamped_layer_of_one_token(zlib, oracle, dev, fused):
    """the one-kernel form: the bits of the separate launches, which the oracle pins above"""
    import torch
    w, x, _, _, clamp, _ = _layer(zlib, oracle, dev, synth.Q4_K, 1, fused, 89)
    rng = synth.rng_for(90)
    ctx = zlib.Context(1, D, F, E, K)
    layer = zlib.Layer(ctx, D, F, E, K, (synth.Q4_K,) * 3, *[to_dev(a, dev) for a in w], clamp=clamp, clamp_fused=fused,
                       router_w=to_dev(synth.router_weights(E, D, rng, sigma=D ** -0.5), dev))
    xd, n0 = to_dev(x, dev), zlib.load().zmoe_kernel_launches()
    one, sep = torch.empty((1, D), device=dev), torch.empty((1, D), device=dev)
    layer.forward(xd, one)
    assert zlib.load().zmoe_kernel_launches() == n0 + 1
    act = ctx.act(K, F).copy()
    layer.route(xd)
    layer.expert_ffn(sep)
    torch.cuda.synchronize()
    ctx.check()
    assert np.array_equal(one.cpu().numpy().view(np.uint32), sep.cpu().numpy().view(np.uint32))
    assert np.array_equal(act.view(np.uint32), ctx.act(K, F).view(np.uint32))
