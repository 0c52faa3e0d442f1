"""GPU parity of the few-token kernels of linear_skinny.cu (fp16, 2..27 tokens, Q4_K and Q6_K) at the edges of their
ranges: token groups of eight, row tiles of sixteen (a gate/up pair: eight), the row counts from which a CTA walks its tiles
with two and four row groups and in several passes (17 tokens and more), and the kernel that keeps the tokens in registers
(up to sixteen tokens, more than two tiles per SM, rows of up to 32 super-blocks, odd numbers of them among these)."""

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


def _product(x, deq):
    """x deq^T in 64 bits (on the GPU: the large cases take the CPU seconds)."""
    return (_dev(x).double() @ _dev(deq).double().T).cpu().numpy()


def _rows(tiles_per_sm, tile, extra):
    """Output rows of `tiles_per_sm` tiles on every SM, and some more."""
    return tiles_per_sm * torch.cuda.get_device_properties(0).multi_processor_count * tile + extra


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


@pytest.mark.parametrize("k", [256, 1024, 1280, 1792, 2048, 2304, 3072, 4096, 5120, 7936, 8192])
def test_tokens_in_registers(k):
    """More than two tiles per SM: every width the register kernel takes at its first and last warp counts, one and two
    super-blocks per warp, whole and with a half-empty last warp.  The rows' padding holds bytes that decode to NaN."""
    rng = np.random.default_rng([k, 7])
    n = _rows(2, 16, 7)
    w, deq = _weights("q4_k", rng, n, k)
    padded = torch.full((n, w.shape[1] + 48), 0xFF, dtype=torch.uint8, device=DEV)
    padded[:, :w.shape[1]] = _dev(w)
    for m in (2, 8, 9, 16):
        x, res = synth.activations(rng, m, k), synth.activations(rng, m, n)
        y = torch.ops.alloy.gguf_q4_k_mm(_dev(x), _dev(w))
        assert_close(to_np(y), _product(x, deq), torch.float16, f"{m}x{n}x{k}")
        assert torch.equal(torch.ops.alloy.gguf_q4_k_mm(_dev(x), padded[:, :w.shape[1]]), y)
        yr = torch.ops.alloy.linear_residual(_dev(x), _dev(w), None, _dev(res), "q4_k")
        assert torch.equal(yr, (_dev(res).float() + y.float()).half())
        # the same rows as three matrices of one launch, ragged
        cuts = [0, 37, n // 2 + 3, n]
        parts = ops.linear_multi(_dev(x), [("q4_k", _dev(w[lo:hi]), None) for lo, hi in zip(cuts, cuts[1:])])
        assert torch.equal(torch.cat(parts, 1), y)
        g = n - 3
        xg = (x.astype(np.float32) * 3 / np.sqrt(k)).astype(np.float16)
        yg = torch.ops.alloy.gguf_q4_k_silu(_dev(xg), _dev(w[:g]), _dev(w[n - g:]))
        r = _product(xg, deq)
        assert_close(to_np(yg), O.silu(r[:, :g]) * r[:, n - g:], torch.float16, f"gated {m}x{g}x{k}")
    assert _lib.load().alloyb_device_error(1) == 0


@pytest.mark.parametrize("fmt,tiles,extra,k", [("q4_k", 6, 131, 512), ("q4_k", 17, 5, 256), ("q6_k", 2, 9, 2048), ("q6_k", 10, 321, 2048)])
def test_row_groups_and_passes(fmt, tiles, extra, k):
    """17 tokens and more: two and four row groups, several passes over K, rings that run on from pass to pass; dense rows and
    rows with padding."""
    rng = np.random.default_rng([tiles, k])
    n = _rows(tiles, 16, extra)
    w, deq = _weights(fmt, rng, n, k)
    op = torch.ops.alloy.gguf_q4_k_mm if fmt == "q4_k" else torch.ops.alloy.gguf_q6_k_mm
    padded = torch.full((n, w.shape[1] + 48), 0xFF, dtype=torch.uint8, device=DEV)
    padded[:, :w.shape[1]] = _dev(w)
    for m in (17, 24, 27):
        x = synth.activations(rng, m, k)
        y = op(_dev(x), _dev(w))
        assert_close(to_np(y), _product(x, deq), torch.float16, f"{fmt} {m}x{n}x{k}")
        assert torch.equal(op(_dev(x), padded[:, :w.shape[1]]), y)
    assert _lib.load().alloyb_device_error(1) == 0


@pytest.mark.parametrize("tiles,extra", [(5, 1), (8, 129), (18, 3)])
def test_row_groups_and_passes_gated(tiles, extra):
    rng = np.random.default_rng([tiles, 2])
    n, k = _rows(tiles, 8, extra), 512
    (g, gd), (u, ud) = _weights("q4_k", rng, n, k), _weights("q4_k", rng, n, k)
    for m in (17, 24, 27):
        x = (synth.activations(rng, m, k, np.float32) * 3 / np.sqrt(k)).astype(np.float16)
        y = torch.ops.alloy.gguf_q4_k_silu(_dev(x), _dev(g), _dev(u))
        assert_close(to_np(y), O.silu(_product(x, gd)) * _product(x, ud), torch.float16, f"gated {m}x{n}x{k}")
    assert _lib.load().alloyb_device_error(1) == 0


@pytest.mark.parametrize("tiles", [(2, 1, 1), (5, 0, 3)])
def test_row_groups_over_mixed_matrices(tiles):
    """Passes end where a matrix ends: Q4_K and Q6_K stages of different sizes in one ring, row groups without a tile."""
    rng = np.random.default_rng(tiles)
    k, fmts = 2048, ("q4_k", "q4_k", "q6_k")
    mats = [(fmt, *_weights(fmt, rng, _rows(t, 16, 16 + 3 * i), k)) for i, (fmt, t) in enumerate(zip(fmts, tiles))]
    for m in (17, 24, 27):
        x = synth.activations(rng, m, k)
        for y, (fmt, _, deq) in zip(ops.linear_multi(_dev(x), [(f, _dev(w), None) for f, w, _ in mats]), mats):
            assert_close(to_np(y), _product(x, deq), torch.float16, f"mixed {fmt} {m} {tiles}")
    assert _lib.load().alloyb_device_error(1) == 0


@pytest.mark.parametrize("m", [5, 16, 17, 27])
@pytest.mark.parametrize("k", [2048, 4096, 8192])
@pytest.mark.parametrize("scale", [60000.0, 1e-4])
def test_few_tokens_extreme_activations(scale, k, m):
    """The sums of x enter the minima's product in two pieces scaled to fit any activations: at both ends of fp16's range
    the error stays that of the output's rounding.  (More than two tiles per SM: the kernels of linear_skinny.cu.)"""
    rng = np.random.default_rng(9)
    n = _rows(2, 16, 7)
    w = synth.q4k_blocks(rng, n, k)
    x = (rng.uniform(0.5, 1.0, (m, k)) * scale).astype(np.float16)
    deq = O.dequant_q4_k(w)
    # only the first four are not zero among the large ones: their sum is past fp16's range, many outputs are not
    if scale > 1:
        x[:, 4:] = 0
    ref = _product(x, deq)
    keep = np.abs(ref) < 6e4
    y = to_np(torch.ops.alloy.gguf_q4_k_mm(_dev(x), _dev(w))).astype(np.float64)
    bound = 2.0 ** -10 * np.abs(ref) + 2.0 ** -20 * _product(np.abs(x), np.abs(deq)) + 2.0 ** -24
    assert keep.any() and (np.abs(y - ref)[keep] <= bound[keep]).all()


@pytest.mark.parametrize("k", [2048, 4096, 7936])
@pytest.mark.parametrize("m", [4, 16, 27])
def test_few_tokens_that_cancel(k, m):
    """Tokens whose products with a row cancel to almost nothing leave the error of the sums alone: K / 16 products of the
    tensor core and their additions, each to 2^-23 of what has come together, which stays below a few times sqrt(sum |w x|^2)
    -- 2^-22 of sum |w x| is past all of it.  (Measured: 2^-24 at most; the kernel of linear_mma.cu, 2^-21.)"""
    rng = np.random.default_rng([k, m])
    n = _rows(2, 16, 7)
    w = synth.q4k_blocks(rng, 1, k)
    row = O.dequant_q4_k(w)[0].astype(np.float64)
    x = synth.activations(rng, m, k)
    for i in range(m):
        at = rng.choice(np.argsort(-np.abs(row))[:k // 4], 4, replace=False)
        x[i, at] = 0
        for j in at:                        # each takes up what the rounding of the one before has left
            x[i, j] = np.float16(-(x[i].astype(np.float64) @ row) / row[j])
    y = to_np(torch.ops.alloy.gguf_q4_k_mm(_dev(x), _dev(np.repeat(w, n, 0)))).astype(np.float64)
    ref, mag = x.astype(np.float64) @ row, np.abs(x.astype(np.float64)) @ np.abs(row)
    if k <= 4096 or m <= 8 or m > 16:       # (the others go to linear_mma.cu)
        assert (np.abs(y - ref[:, None]) <= 2.0 ** -22 * mag[:, None] + 2.0 ** -11 * np.abs(ref[:, None])).all()


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
        # (one token against Q4_K: the norm runs inside the streaming kernel, with a rounding less)
        assert all(torch.equal(p, q) for p, q in list(zip(a, b))[2 if m == 1 else 0:])
