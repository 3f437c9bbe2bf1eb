"""Attention over smooth slot states (half-lives long against a 128-step tile) against the every-step fp32 kernels on the
same 16-bit inputs.

Tolerances (norm-wise, helpers.rel_err).  u = 2^-11 is the rounding of a 16-bit operand; an output term passes five such operands
(state, W_pe, gate coefficient, E row, probability), and its probability moves by 5 u times the score on top: with the E rows of
std 0.1 used here scores stay near one, 10 u = 5e-3.  Gradients: the hot slots of every tile come from the every-step kernel, in
bf16, so the 2e-2 that the suite allows that kernel.
"""
import numpy as np
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu

TOL_O, TOL_GRAD = 5e-3, 2e-2


@pytest.fixture(scope="module")
def mb():
    import mathbrain_b200 as m
    m._lib.load()
    m.set_options(inactive_mass="full_V", cbase_extra_decay=False, mode="fp32")
    return m


def case(seed, T, K, N, H=2, B=2, min_hl=1024.0, std=0.02, fill=None, dtype=torch.bfloat16, state=50.0, unlisted=float("nan")):
    """Lists of K slots (sample 0) and of about half (later samples, the first entry unlisted); the E rows of unlisted
    entries hold anything."""
    g = torch.Generator().manual_seed(seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    D, V = 64 * H, max(2000, 2 * K)
    unique = torch.full((B, K), -1, dtype=torch.long)
    x = torch.zeros(B, T, dtype=torch.long)
    for b in range(B):
        n = K if b == 0 else max(1, K // 2)
        lo = 0 if b == 0 or K == 1 else 1
        toks = rng.permutation(V)[:n]
        unique[b, lo:lo + n] = torch.from_numpy(toks)[:K - lo]
        listed = unique[b][unique[b] >= 0].numpy()
        # half the steps take listed tokens, those near the front of the list again and again
        pick = listed[np.minimum((rng.random(T) ** 3 * len(listed)).astype(int), len(listed) - 1)]
        x[b] = torch.from_numpy(np.where(rng.random(T) < 0.5, pick, rng.integers(0, V, T)))
    rhos = torch.exp(-np.log(2.0) / torch.logspace(np.log10(min_hl), np.log10(4 * min_hl), N))
    r = lambda *s, std=std: torch.randn(*s, generator=g) * std
    # at least a tenth of a slot's size: far smaller states make the operand products subnormal in fp16, with roundings above u
    c_base = (0.1 + 0.9 * torch.rand(B, K, N, generator=g)) * state * (0.02 + 0.98 * torch.rand(B, K, 1, generator=g) ** 4)
    E = [r(B, K, D, std=0.1), r(B, K, D, std=0.1)]
    for e in E:
        e[unique < 0] = unlisted
    d = dict(x=x, unique=unique, rhos=rhos, c_base=c_base, Q=r(B, H, T, 64, std=1.0).to(dtype), Ek=E[0].to(dtype), Ev=E[1].to(dtype),
             W=r(N, D), dO=r(B, H, T, 64, std=1.0), fill=None if fill is None else torch.tensor(fill, dtype=torch.int32))
    if fill is not None:
        for b, n in enumerate(fill):
            d["dO"][b, :, n:] = 0
    return {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in d.items()}, V


def attend(mb, c, V, mode, silu=True, rows=None):
    with mb.options(mode=mode):
        h = mb.precompute_boundaries(c["x"], c["unique"], c["rhos"], 64, c_init=c["c_base"], seq_lens=c["fill"])
        Q, Ek, Ev, W = (c[k].clone().requires_grad_(True) for k in ("Q", "Ek", "Ev", "W"))
        K = c["unique"].shape[1]
        if rows is None:
            O = mb.FlashEMAFunction.apply(Q, c["x"], Ek, Ev, W, c["rhos"], V, c["unique"], K, h, silu)
        else:
            O = mb.FlashEMARowsFunction.apply(Q, c["x"], Ek, Ev, rows, W, c["rhos"], V, c["unique"], K, h, silu)
        O.backward(c["dO"])
    assert mb.device_status() == 0
    return dict(O=O.detach(), dQ=Q.grad, dEk=Ek.grad, dEv=Ev.grad, dW=W.grad)


def compare(out, ref):
    for k in out:
        assert rel_err(out[k].float(), ref[k].float()) < (TOL_O if k == "O" else TOL_GRAD), k


def compare_rows(out, ref, names=("dEk", "dEv", "dQ"), floor=1e-3):
    """Every row against its own size (2-norm), down to `floor` of the largest row: the largest rows are the hot slots', which the
    every-step kernel makes, many times the size of the others."""
    for k in names:
        a, b = out[k].double().flatten(0, -2), ref[k].double().flatten(0, -2)
        assert bool(torch.isfinite(a).all()), k
        n = b.norm(dim=1)
        live = n > floor * n.max()
        err = ((a - b).norm(dim=1) / n)[live]
        assert float(err.max()) < TOL_GRAD, (k, float(err.max()))


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("T,K", [(1, 1), (127, 17), (128, 16), (129, 144), (130, 145), (300, 400), (513, 1100)])
def test_edges_of_tiles_and_item_blocks(mb, N, T, K):
    c, V = case(T + K, T, K, N)
    compare(attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32"))


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("min_hl", [512.0, 200.0, 100.0, 50.0, 5.0])
def test_segments_of_faster_decays(mb, N, min_hl):
    """One, two, four and eight segments in the forward; up to eight and every step in the backward."""
    c, V = case(int(min_hl), 260, 300, N, min_hl=min_hl)
    compare(attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32"))


@pytest.mark.parametrize("std", [0.1, 0.4, 2.0])
def test_segments_of_large_pre_activations(mb, std):
    """The change of the pre-activation inside a tile picks the segments, up to every step (std 2)."""
    c, V = case(77, 200, 200, 64, std=std, state=20.0)
    c["Ek"], c["Ev"] = c["Ek"] * 0.1 / std, c["Ev"] * 0.1 / std      # scores stay near one
    compare(attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32"))


@pytest.mark.parametrize("N,H", [(64, 2), (64, 6), (128, 4)])
def test_rows_of_small_gradients(mb, N, H):
    c, V = case(21, 300, 500, N, H=H, unlisted=0.0)
    compare_rows(attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32"), names=("dEk", "dEv"), floor=1e-4)


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("ev", [0.01, 1.0, 30.0])
def test_values_and_gradients_of_any_size_in_a_peaked_softmax(mb, N, ev):
    """Two slots of moderate state (not among the hot ones) share every row's softmax and dO points along the difference of their
    values: |dP - D| is thousands of times max |dO| for ev = 30."""
    c, V = case(8, 300, 200, N, unlisted=0.0, state=20.0)
    listed = c["unique"] >= 0
    pair = torch.tensor([50, 60], device="cuda")
    c["x"] = torch.where((c["x"][..., None] == c["unique"][:, None, pair]).any(-1), c["unique"][:, :1].clamp_min(0), c["x"])
    c["c_base"][:, pair] = 4.0
    c["W"] = c["W"].abs() + 0.01                     # gates of one sign
    c["Q"] = torch.ones_like(c["Q"]) * 0.5
    c["Ek"] = torch.zeros_like(c["Ek"])
    scale = 16.0 / (4.0 * float(c["W"].sum(0).mean()) * 64 * 0.5 / 8)
    c["Ek"][:, pair] = scale
    c["Ek"][:, pair[1], ::2] *= 1.5                  # (equal keys would cancel in dQ)
    c["Ek"][:, pair[1], 1::2] *= 0.5
    g = torch.Generator().manual_seed(2)
    c["Ev"] = ((torch.randn(c["Ev"].shape, generator=g) * ev).cuda() * listed[..., None]).to(c["Ev"].dtype)
    d = torch.sign(c["Ev"][:, pair[0]].float() - c["Ev"][:, pair[1]].float())
    c["dO"] = d.view(d.shape[0], -1, 1, 64).expand(-1, -1, c["x"].shape[1], -1).contiguous() * 0.01
    out, ref = attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32")
    compare_rows(out, ref)
    assert rel_err(out["dW"], ref["dW"]) < TOL_GRAD


@pytest.mark.parametrize("N", [64, 128])
def test_gradient_rows_of_very_different_size(mb, N):
    """A row of dO smaller by a power of two gives the row of dQ smaller by it, whatever stands beside it in the tile."""
    c, V = case(41, 300, 300, N, unlisted=0.0)
    plain = attend(mb, c, V, "tc_bf16")
    f = 2.0 ** -torch.randint(0, 60, c["dO"].shape[:3], generator=torch.Generator().manual_seed(4)).float().cuda()[..., None]
    c["dO"] = c["dO"] * f
    c["Q"] = c["Q"].float()                # dQ in fp32
    out, ref = attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32")
    compare(out, ref)
    a, b = (out["dQ"] / f).double().flatten(0, -2), plain["dQ"].double().flatten(0, -2)
    assert float(((a - b).norm(dim=1) / b.norm(dim=1)).max()) < 2.0 ** -7      # `plain` is rounded to bf16


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_gradients_that_are_not_finite_say_so(mb, bad):
    c, V = case(43, 300, 300, 64, H=4, unlisted=0.0)
    c["dO"][1, 2, 150, 7] = bad
    out = attend(mb, c, V, "tc_bf16")
    finite = {k: torch.isfinite(v) for k, v in out.items()}
    rows = finite["dQ"].all(-1)
    assert not bool(rows[1, 2, 150]) and int((~rows).sum()) == 1
    listed = (c["unique"][1] >= 0)
    for k in ("dEk", "dEv"):
        heads = finite[k].view(*finite[k].shape[:2], 4, 64)
        assert not bool(heads[1, listed, 2].all(-1).any())
        heads[1, :, 2] = True
        assert bool(heads.all())
    assert not bool(finite["dW"].view(64, 4, 64)[:, 2].all()) and bool(finite["dW"].view(64, 4, 64)[:, [0, 1, 3]].all())


def test_columns_of_unequal_size(mb):
    """Eight columns of W_pe fifteen times the others, of opposite signs on fast and slow channels, so that their pre-activations pass
    through zero inside the tile, by some 8 either way; the root mean square over all columns is near 1.  Every column of the output against its own size:
    the roundings of state and W_pe (u/2 each) leave 0.4 u |M W|_2 = 0.4 u 120 in a pre-activation, 7e-3 of a gate of some 4."""
    c, V = case(51, 256, 200, 64, H=8, unlisted=0.0)
    c["c_base"] = 50.0 + 4.0 * torch.rand(c["c_base"].shape, generator=torch.Generator().manual_seed(1)).cuda()
    mid = c["rhos"] ** 63.5
    fast = c["rhos"] < c["rhos"].median()
    w = torch.where(fast, -0.3, 0.3 * float(mid[fast].sum() / mid[~fast].sum()))
    cols = torch.arange(8, device="cuda") * 64 + 5
    c["W"][:, cols] = w[:, None] * torch.tensor([1.0, -1.0] * 4, device="cuda")
    out, ref = attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32")
    a, b = (o["O"].double().permute(0, 2, 1, 3).flatten(0, 1).flatten(1) for o in (out, ref))
    n = b.norm(dim=0)
    err = (a - b).norm(dim=0) / n.clamp_min(1e-3 * float(n.max()))      # (columns whose gates are all far below zero are rounding alone)
    assert float(err.max()) < 1.5e-2, (float(err[cols].max()), float(err.max()))


@pytest.mark.parametrize("silu,dtype", [(False, torch.bfloat16), (True, torch.float32)])
def test_linear_gate_and_fp32_inputs(mb, silu, dtype):
    c, V = case(5, 257, 333, 64, dtype=dtype)
    compare(attend(mb, c, V, "tc_bf16", silu), attend(mb, c, V, "fp32", silu))


def test_ragged_batch(mb):
    c, V = case(9, 400, 300, 64, B=4, fill=[400, 129, 128, 0])
    out, ref = attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32")
    compare(out, ref)
    for b, n in enumerate([400, 129, 128, 0]):
        assert float(out["O"][b, :, n:].abs().sum()) == 0.0 and float(out["dQ"][b, :, n:].float().abs().sum()) == 0.0


@pytest.mark.parametrize("N", [64, 128])
def test_shared_rows(mb, N):
    """Rows shared between the samples, the hot slots at every step in both directions; unlisted entries point to a row of
    their own that holds NaN."""
    c, V = case(31, 300, 250, N, unlisted=0.0)
    tokens, index = mb.shared_slot_rows(c["unique"])
    U, D = tokens.numel(), c["W"].shape[1]
    index[c["unique"] < 0] = U
    g = torch.Generator().manual_seed(1)
    for k in ("Ek", "Ev"):
        c[k] = torch.cat([torch.randn(U, D, generator=g) * 0.1, torch.full((1, D), float("nan"))]).bfloat16().cuda()
    out, ref = attend(mb, c, V, "tc_bf16", rows=index), attend(mb, c, V, "fp32", rows=index)
    compare(out, ref)


def test_states_of_the_fp32_mode_serve_the_tensor_core_mode(mb):
    """Snapshots taken in the fp32 mode carry no items: the operator builds them itself, with the same result."""
    c, V = case(3, 200, 150, 64)
    res = []
    for first in ("tc_bf16", "fp32"):
        with mb.options(mode=first):
            h = mb.precompute_boundaries(c["x"], c["unique"], c["rhos"], 64, c_init=c["c_base"])
        with mb.options(mode="tc_bf16"):
            Q = c["Q"].clone().requires_grad_(True)
            O = mb.FlashEMAFunction.apply(Q, c["x"], c["Ek"], c["Ev"], c["W"], c["rhos"], V, c["unique"], c["unique"].shape[1], h, True)
            O.backward(c["dO"])
        res.append((O.detach(), Q.grad))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


def test_bounded_waits_give_up_cleanly(mb):
    """The first arrival of the gate warps is withheld by the library's test hook: the launch ends by itself and the status
    names a wait; after clear_status() results are right again (all tensor memory was given back)."""
    c, V = case(13, 200, 300, 64)
    mb.ops.clear_status()
    mb.ops._OPTIONS["_test_withhold_arrive"] = True
    try:
        with mb.options(mode="tc_bf16"), torch.no_grad():
            h = mb.precompute_boundaries(c["x"], c["unique"], c["rhos"], 64, c_init=c["c_base"])
            mb.FlashEMAFunction.apply(c["Q"], c["x"], c["Ek"], c["Ev"], c["W"], c["rhos"], V, c["unique"], c["unique"].shape[1], h, True)
    finally:
        mb.ops._OPTIONS["_test_withhold_arrive"] = False
    torch.cuda.synchronize()
    assert mb.device_status() & 1
    mb.ops.clear_status()
    compare(attend(mb, c, V, "tc_bf16"), attend(mb, c, V, "fp32"))


@pytest.mark.parametrize("mode", ["tc_bf16", "fp32"])
def test_empty_batch(mb, mode):
    c, V = case(3, 130, 40, 64)
    for k in ("x", "unique", "c_base", "Q", "Ek", "Ev", "dO"):
        c[k] = c[k][:0]
    out = attend(mb, c, V, mode)
    assert out["O"].shape == c["Q"].shape and float(out["dW"].abs().max()) == 0.0
