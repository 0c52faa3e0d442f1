"""GPU parity of the few-token kernels of linear_skinny.cu (fp16, 2..27 tokens, Q4_K and Q6_K) at the edges of their
ranges: token groups of eight, row tiles of sixteen (a gate/up pair: eight), the K widths whose token fragments live in
registers (2048, 4096, 8192 up to sixteen tokens) and the others."""

import numpy as np
import pytest
import torch

from alloy_b200 import _lib, ops, synth
from oracle import blocks as O
from tests._util import assert_close, to_np

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _weights(fmt, rng, n, k):
    w = (synth.q4k_blocks if fmt == "q4_k" else synth.q6k_blocks)(rng, n, k)
    return w, (O.dequant_q4_k if fmt == "q4_k" else O.dequant_q6_k)(w)


@pytest.mark.parametrize("fmt,n,k", [("q4_k", 40, 2048), ("q4_k", 1000, 4096), ("q4_k", 33, 8192), ("q4_k", 77, 768),
                                     ("q4_k", 4800, 2048), ("q6_k", 40, 2048), ("q6_k", 520, 14336)])
@pytest.mark.parametrize("m", [2, 8, 9, 16, 17, 24, 25, 27])
def test_few_tokens(fmt, n, k, m):
    rng = np.random.default_rng([n, k, m])
    w, deq = _weights(fmt, rng, n, k)
    x, res = synth.activations(rng, m, k), synth.activations(rng, m, n)
    ref = x.astype(np.float64) @ deq.astype(np.float64).T
    y = (torch.ops.alloy.gguf_q4_k_mm if fmt == "q4_k" else torch.ops.alloy.gguf_q6_k_mm)(_dev(x), _dev(w))
    assert_close(to_np(y), ref, torch.float16, f"{fmt} {m}x{n}x{k}")
    # residual: half(residual + half(acc)), the first rounding being the one compared above
    yr = torch.ops.alloy.linear_residual(_dev(x), _dev(w), None, _dev(res), fmt)
    assert torch.equal(yr, (_dev(res).float() + y.float()).half())
    assert _lib.load().alloyb_device_error(1) == 0


@pytest.mark.parametrize("n,k", [(44, 2048), (2400, 4096), (13, 8192), (50, 1280)])
@pytest.mark.parametrize("m", [3, 8, 12, 16, 20, 27])
def test_few_tokens_gated(n, k, m):
    rng = np.random.default_rng([n, k, m, 1])
    (g, gd), (u, ud) = _weights("q4_k", rng, n, k), _weights("q4_k", rng, n, k)
    x = (synth.activations(rng, m, k, np.float32) * 3 / np.sqrt(k)).astype(np.float16)
    x64 = x.astype(np.float64)
    for op, act in ((torch.ops.alloy.gguf_q4_k_silu, O.silu), (torch.ops.alloy.gguf_q4_k_gelu, O.gelu_tanh)):
        assert_close(to_np(op(_dev(x), _dev(g), _dev(u))), act(x64 @ gd.T.astype(np.float64)) * (x64 @ ud.T.astype(np.float64)),
                     torch.float16, f"gated {m}x{n}x{k}")


@pytest.mark.parametrize("m", [4, 16, 23])
def test_few_tokens_mixed_formats(m):
    rng = np.random.default_rng([m, 5])
    k, specs, refs = 4096, [], []
    x = synth.activations(rng, m, k)
    for fmt, n in (("q4_k", 200), ("q4_k", 64), ("q6_k", 72)):
        w, deq = _weights(fmt, rng, n, k)
        specs.append((fmt, _dev(w), None))
        refs.append(x.astype(np.float64) @ deq.astype(np.float64).T)
    for y, ref in zip(ops.linear_multi(_dev(x), specs), refs):
        assert_close(to_np(y), ref, torch.float16, f"mixed {m}")


@pytest.mark.parametrize("scale", [60000.0, 1e-4])
def test_few_tokens_extreme_activations(scale):
    """The sums of x enter the minima's product in two pieces scaled to fit any activations: at both ends of fp16's range
    the error stays that of the output's rounding."""
    rng = np.random.default_rng(9)
    n, k, m = 48, 2048, 5
    w = synth.q4k_blocks(rng, n, k)
    x = (rng.uniform(0.5, 1.0, (m, k)) * scale).astype(np.float16)
    deq = O.dequant_q4_k(w).astype(np.float64)
    # only the first four are not zero among the large ones: their sum is past fp16's range, many outputs are not
    if scale > 1:
        x[:, 4:] = 0
    ref = x.astype(np.float64) @ deq.T
    keep = np.abs(ref) < 6e4
    y = to_np(torch.ops.alloy.gguf_q4_k_mm(_dev(x), _dev(w))).astype(np.float64)
    bound = 2.0 ** -10 * np.abs(ref) + 2.0 ** -20 * (np.abs(x).astype(np.float64) @ np.abs(deq).T) + 2.0 ** -24
    assert keep.any() and (np.abs(y - ref)[keep] <= bound[keep]).all()


@pytest.mark.parametrize("m", [1, 4, 16, 24])
def test_tokens_that_the_launch_before_has_just_written(m):
    """The normalised tokens come from the launch right before: read behind the wait, never ahead of it.  Calls queued back
    to back, each on other tokens, against calls that are waited for one by one."""
    gen = torch.Generator(device=DEV).manual_seed(m)
    n, k = 2 * torch.cuda.get_device_properties(0).multi_processor_count * 16 + 16, 4096
    g, u = (synth.q4k_blocks_device(n, k, gen) for _ in range(2))
    q8 = synth.q8_0_weight_device(n, k, gen)
    w = torch.rand(k, device=DEV, generator=gen).half()
    xs = [torch.randn((m, k), device=DEV, generator=gen).half() for _ in range(6)]

    def calls(x):
        return [ops.gated_normed(x, w, 1e-5, g, u), *ops.linear_multi(x, [("q4_k", g, None)], norm=(w, 1e-5)),
                *ops.linear_multi(x, [("q8_0", *q8)], norm=(w, 1e-5))]

    want = []
    for x in xs:
        xn = ops.rms_norm(x, w, 1e-5)
        torch.cuda.synchronize()
        want.append([torch.ops.alloy.gguf_q4_k_silu(xn, g, u), torch.ops.alloy.gguf_q4_k_mm(xn, g), torch.ops.alloy.gguf_q8_0_mm(xn, *q8)])
        torch.cuda.synchronize()
    for a, b in zip([calls(x) for x in xs], want):
        assert all(torch.equal(p, q) for p, q in zip(a, b))
