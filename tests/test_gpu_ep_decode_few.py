"""Expert-parallel decode on the sides of the lines up to which values are their own arrival flags: shards with pairs held
elsewhere, a shard that none of the tokens chose, and the peer exchange with a world of one rank."""
from types import SimpleNamespace

import numpy as np
import pytest

from fngine_b200 import lib as L
from fngine_b200 import synth

pytestmark = pytest.mark.gpu
H = 2560
IQ3_S, IQ4_NL = L.FMT_IQ3_S, L.FMT_IQ4_NL
CASES = ([(IQ3_S, IQ3_S, 512, t) for t in (1, 2, 3, 4)] + [(IQ4_NL, IQ4_NL, 512, t) for t in (1, 4, 16)] +
         [(IQ3_S, IQ4_NL, 640, t) for t in (1, 2)])


def _setup(fg, fd, inter, tokens, seed):
    import torch
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    from fngine_b200 import moe
    full = moe.synth_layer(fg, fd, inter, 512, seed)
    wr = torch.from_numpy(synth.router_weights(303, rows=512).view(np.int16)).cuda().view(torch.bfloat16)
    x = torch.from_numpy(synth.activations(90 + tokens, tokens)).cuda()
    return torch, moe, full, wr, x, moe.DecodeWorkspace(full)


@pytest.mark.parametrize("fg,fd,inter,tokens", CASES)
def test_shards_of_few_tokens(fg, fd, inter, tokens):
    """Three ranks played one after another on one workspace: the even and the odd experts that were chosen, and a rank
    whose experts nobody chose. The sum of the partial rows is the layer (the ranks' sums are added in another order than one
    rank's pairs: fp32 rounding), the third rank's rows are zero."""
    torch, moe, full, wr, x, ws = _setup(fg, fd, inter, tokens, 5100)
    from fngine_b200 import ep
    y = torch.empty(tokens, H, dtype=torch.float32, device="cuda")
    moe.moe_layer_decode(wr, full, x, ws, y)
    torch.cuda.synchronize()
    chosen = sorted(set(np.asarray(ws.work().topk_expert)[:tokens].reshape(-1).tolist()))
    idle = [e for e in range(512) if e not in chosen][:7]
    parts = torch.full((3, tokens, H), float("nan"), dtype=torch.float32, device="cuda")
    for call in range(2):  # (the second time, other activations over what the first one left in the workspace)
        held = 0
        for r, experts in enumerate([chosen[0::2], chosen[1::2], idle]):
            slots = np.full(512, -1, np.int32)
            slots[experts] = np.arange(len(experts), dtype=np.int32)
            shard = SimpleNamespace(layer=moe.synth_layer_of(fg, fd, inter, experts, 5100),
                                    slot_of=torch.from_numpy(slots).cuda())
            ep.layer_decode_ep(wr, shard, x if call == 0 else 0.75 * x, ws, parts[r])
            torch.cuda.synchronize()
            work = ws.work()
            assert ws.status() == 0 and work.n_cold == 10 * tokens - work.n_pairs
            assert all(work.token_pair_count[t] + work.token_cold_count[t] == 10 for t in range(tokens))
            held += work.n_pairs
        if call == 0:
            assert held == 10 * tokens and bool((parts[2] == 0.0).all())
            got = ep.combine_sum(parts)
            err = torch.linalg.vector_norm(got - y, dim=1) / torch.linalg.vector_norm(y, dim=1)
            assert float(err.max()) <= 1e-6
    assert bool(torch.isfinite(parts).all())


@pytest.mark.parametrize("fg,fd,inter,tokens", CASES)
def test_peer_exchange_of_few_tokens_with_one_rank(fg, fd, inter, tokens):
    """The rank is its own peer (nobody else is waited for): the plain layer's bits, on both buffer parities."""
    torch, moe, full, wr, x, ws = _setup(fg, fd, inter, tokens, 5200)
    from fngine_b200 import ep
    lib = L.load()
    bufs = [torch.zeros(lib.fb_ep_exchange_bytes(k), dtype=torch.uint8, device="cuda") for k in (0, 1)]
    xchg = SimpleNamespace(rank=0, world=1, step=0, peers=L.EpPeers())
    xchg.peers.rank, xchg.peers.n_ranks = 0, 1
    xchg.peers.x_all[0], xchg.peers.y_parts[0] = (b.data_ptr() for b in bufs)
    shard = SimpleNamespace(layer=full, slot_of=torch.arange(512, dtype=torch.int32, device="cuda"))
    y, want = (torch.empty(tokens, H, dtype=torch.float32, device="cuda") for _ in range(2))
    for step in range(3):
        xs = x + 0.125 * step
        moe.moe_layer_decode(wr, full, xs, ws, want)
        y.fill_(float("nan"))
        ep.layer_decode_ep_p2p(wr, shard, xs, ws, xchg, y)
        torch.cuda.synchronize()
        assert ws.status() == 0 and torch.equal(y, want)
