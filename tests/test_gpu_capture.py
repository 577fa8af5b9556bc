"""Batched device calls inside a captured graph: the job tables are the
graph's own, so a replay gives the call's results whatever became of the host
memory they were made in."""
import numpy as np
import pytest
import torch

import pcg_b200 as L

pytestmark = pytest.mark.gpu


def words(rng, n):
    return torch.from_numpy(rng.integers(0, L.P, n, dtype=np.uint64).view(np.int64)).cuda()


def stream():
    return torch.cuda.current_stream().cuda_stream


def products(rng):
    lens = [1 << 16, 1 << 18, 1 << 17]
    a, b = ([words(rng, n) for n in lens] for _ in range(2))
    c = [torch.zeros_like(v) for v in a]
    vp = L.C.c_void_p

    def call():
        ptrs = [(vp * 3)(*[v.data_ptr() for v in q]) for q in (c, a, b)]
        rc = L.lib.pcgb_poly_mul_device_multi(3, *ptrs, (L.C.c_int * 3)(*lens), stream())
        assert rc == 0, L.lib.pcgb_last_error()
    return call, a + b, c


def key_groups(rng):
    groups, ins, outs = [], [], []
    for K, n in ((64, 9), (300, 14), (5, 16)):
        r, cw = words(rng, 2 * K), words(rng, 2 * K * n)
        out = torch.zeros(2 * K << n, dtype=torch.int64, device="cuda")
        groups.append((K, n, r.data_ptr(), cw.data_ptr(), out.data_ptr()))
        ins += [r, cw]
        outs.append(out)
    return (lambda: L.dpf_keyed_full_eval_multi_device(groups, 1, L.PRG_CHACHA8, stream=stream()),
            ins, outs)


def expansions(rng):
    reqs, ins, outs = [], [], []
    for N, c, t in ((1 << 14, 2, 8), (1 << 16, 2, 8)):
        e = L.Expander(N, c, t, 1, L.PRG_CHACHA8, public_a=L.public_a(N, c, 7))
        e.set_leaf_shape(64, 8)
        pos, val = L.noise(N, c, t, 1, 0)
        k = [words(rng, 2 * e.K), words(rng, 2 * e.K * e.levels), words(rng, e.K),
             torch.from_numpy(pos.view(np.int64)).cuda(), torch.from_numpy(val.view(np.int64)).cuda()]
        o = [torch.zeros(N, dtype=torch.int64, device="cuda") for _ in range(2)]
        reqs.append((e, 0, *[v.data_ptr() for v in k + o]))
        ins += k
        outs += o
    return lambda: L.expand_batch_device(reqs, stream()), ins, outs


@pytest.mark.parametrize("make", [products, key_groups, expansions])
def test_replays_own_their_tables(pcg, make):
    call, ins, outs = make(np.random.default_rng(17))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        call()
    torch.cuda.synchronize()
    want = [o.clone() for o in outs]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for size in (64, 400, 3000, 40000, 200000):   # what the tables' heap blocks hold now
        junk = [bytearray(b"\x00" * size) for _ in range(50)]
        for o in outs:
            o.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, w) for o, w in zip(outs, want))
        del junk
    del graph
    torch.cuda.synchronize()
