"""Peer-pull context-parallel attention as rank 1 of 2 on one GPU: the peers' buffers are ordinary tensors of the same
device, the barriers do nothing (no other rank runs), and every result is compared with 64-bit attention."""
import ctypes as C
import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


class _Session:
    """What ``CpSymm`` is to rank 1: a table of both ranks' K, V and staging buffers."""
    world, rank = 2, 1

    def __init__(self, shape, peer_k, peer_v):
        n = math.prod(shape)
        self.own = torch.empty(2, *shape, device="cuda", dtype=torch.bfloat16)
        self.peer = torch.stack([peer_k, peer_v])
        self.stages = torch.full((2, 2, 2, *shape), 7.0, device="cuda")     # [rank][owner][dK | dV]: stale contents
        self.stages[0] = 0                                                 # rank 0 sees none of this rank's keys
        self.slot = 2 * n

    def barrier(self):
        pass

    def kv_buffers(self, key, shape):
        ptrs = [[t[i].data_ptr() for t in (self.peer, self.own)] for i in range(2)]
        return tuple(SimpleNamespace(peer_ptrs=p) for p in ptrs) + (self.own[0], self.own[1])

    def stage(self, shape):
        arr = (C.c_void_p * 2)(*[self.stages[r].data_ptr() for r in range(2)])
        return SimpleNamespace(ptr_array=lambda: arr), self.stages[1], self.slot


@pytest.mark.parametrize("D,Hq,Hkv,L", [(128, 4, 2, 128), (256, 4, 1, 256)])
def test_rank_1_of_2_pulls_the_first_shard(D, Hq, Hkv, L):
    from cverl_b200 import _native as nv
    from cverl_b200.parallel import cp_symm
    g = torch.Generator(device="cuda").manual_seed(D)
    B, n = 2, Hq // Hkv

    def make(h, length):
        return torch.randn(B, h, length, D, device="cuda", generator=g).to(torch.bfloat16)
    q, do = make(Hq, L), make(Hq, L)
    k, v = make(Hkv, 2 * L), make(Hkv, 2 * L)                                # both shards, in order
    first = [t[:, :, :L].transpose(1, 2).contiguous() for t in (k, v)]
    cps = _Session(first[0].shape, *first)
    ctx = SimpleNamespace()
    ctx.save_for_backward = lambda *t: setattr(ctx, "saved_tensors", t)
    out = cp_symm.ring_forward(ctx, q, k[:, :, L:], v[:, :, L:], cps, 0, L, D ** -0.5)
    dq, dk, dv = cp_symm.ring_backward(ctx, do)
    nv.check_status()

    leaves = [t.double().requires_grad_(True) for t in (q, k, v)]
    s = leaves[0] @ leaves[1].repeat_interleave(n, 1).transpose(-1, -2) * D ** -0.5
    s = s.masked_fill(torch.ones(L, 2 * L, dtype=torch.bool, device="cuda").triu(L + 1), float("-inf"))
    want = torch.softmax(s, -1) @ leaves[2].repeat_interleave(n, 1)
    rq, rk, rv = torch.autograd.grad(want, leaves, do.double())
    staged = cps.stages[1, 0].transpose(2, 3)                                # this rank's share for the first shard
    # P, dS, the saved output behind Delta and every hop's result are rounded to bf16, 2^-9 each
    for name, a, r in (("out", out, want), ("dq", dq, rq), ("dk", dk, rk[:, :, L:]), ("dv", dv, rv[:, :, L:]),
                       ("staged dk", staged[0], rk[:, :, :L]), ("staged dv", staged[1], rv[:, :, :L])):
        assert (a.double() - r).norm() <= 5 * 2.0 ** -9 * r.norm(), name
