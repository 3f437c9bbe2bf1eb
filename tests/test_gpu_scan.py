"""Scan and snapshots at the edges of their work split (walked and scanned chains, several long chains a sample, tokens listed twice,
channel counts of every store path), and the row lengths at which the cross-entropy kernels change."""
import numpy as np
import pytest
import torch

from oracle import ema_oracle as orc
from helpers import rel_err

pytestmark = pytest.mark.gpu

TOL_STATE = 1e-5        # fp32 states: a power rounded once per step, a few roundings a step


@pytest.mark.parametrize("T,N,vocab", [(63, 64, 1), (64, 64, 1), (129, 128, 2), (600, 33, 4), (4096, 64, 40), (4096, 128, 300)])
def test_scan_and_snapshots_of_long_chains(T, N, vocab):
    import mathbrain_b200 as mb
    rng = np.random.Generator(np.random.PCG64(T + N))
    B, K = 2, vocab + 3
    x = torch.from_numpy(rng.integers(0, vocab, (B, T)))
    unique = torch.full((B, K), -1, dtype=torch.long)
    for b in range(B):
        unique[b, :vocab] = torch.from_numpy(rng.permutation(vocab))
    unique[:, vocab] = unique[:, 0]                  # a token listed twice, with another state
    unique[0, vocab + 2] = vocab + 5                 # a token that does not occur
    c_base = torch.from_numpy(rng.random((B, K, N)).astype(np.float32) * 40)
    rhos = torch.exp(-np.log(2.0) / torch.logspace(0.3, 3.6, N))
    xd, ud, rd, cd = x.cuda(), unique.cuda(), rhos.cuda(), c_base.cuda()
    C = mb.compute_query_ema_history(xd, rd, vocab + 6, cd, ud)
    assert rel_err(C.cpu(), orc.query_scan(x, rhos, vocab + 6, c_base, unique, dtype=torch.float64)) < TOL_STATE
    h = mb.precompute_boundaries(xd, ud, rd, 64, c_init=cd)
    ref = orc.tile_start_states(x, unique, rhos, 128, c_base, dtype=torch.float64)
    assert rel_err(h.tile_state.cpu(), ref) < TOL_STATE
    n = h.tile_state.numel()
    base = h.tile_state.reshape(-1)
    half = torch.empty(0, dtype=torch.float16, device="cuda").set_(base.untyped_storage(), base.storage_offset() * 2 + 2 * n, (n,))
    assert torch.equal(half.float(), (base / 64).clamp(max=65504.0).half().float())


@pytest.mark.parametrize("V", [24568, 24571, 24576, 57339, 57344, 57345])
def test_cross_entropy_rows_at_the_edges_of_the_shared_memory_path(V):
    import mathbrain_b200 as mb
    lib = mb._lib.load()
    R, ld = 5, (V + 7) // 8 * 8
    g = torch.Generator().manual_seed(V)
    x = (torch.randn(R, ld, generator=g) * 3).bfloat16().cuda()
    t = torch.tensor([0, V - 1, V // 2, -1, V], device="cuda")       # the last two: no target
    loss = torch.empty(R, device="cuda")
    z = x[:, :V].double()
    p = torch.softmax(z, 1)
    want = p.clone()
    want[torch.arange(3), t[:3]] -= 1
    want[3:] = 0
    rc = lib.mbema_ce_rows(x.data_ptr(), 1, t.data_ptr(), 0.5, loss.data_ptr(), R, V, ld, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    ref = (torch.logsumexp(z, 1)[:3] - z[torch.arange(3), t[:3]])
    assert rel_err(loss[:3].cpu(), ref.cpu()) < 1e-6 and float(loss[3:].abs().max()) == 0.0
    assert rel_err(x[:, :V].cpu(), 0.5 * want.cpu()) < 2.0 ** -8            # one rounding to bf16
    assert float(((x[:3, :V].double() - 0.5 * want[:3]).abs() / (0.5 * want[:3].abs())).max()) < 2.0 ** -8 + 1e-5
    assert ld == V or float(x[:, V:].abs().max()) == 0.0
