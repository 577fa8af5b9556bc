"""Outputs over memory that the call has finished reading: x over the keys, z
over the noise, x over the output layers.  Every form gives what separate
buffers give."""
import numpy as np
import pytest

from test_gpu_batch import _request

pytestmark = pytest.mark.gpu


class Request:
    """One expansion's inputs on the host and device buffers to put them in."""

    def __init__(self, pcg, e, seed, party):
        self.pcg, self.e, self.party = pcg, e, party
        (_, _, *ptrs), self.keep = _request(pcg, e, seed, party)
        K, ct = e.K, e.c * e.t
        words = [2 * K, 2 * K * e.levels * e.nk, K, ct, ct]
        bufs = [self.keep[party], *self.keep[2:6]]
        self.host = [b.download(np.uint64, n) for b, n in zip(bufs, words)]
        e.expand_device(party, *ptrs)
        pcg.synchronize()
        self.want = [b.download(np.uint64, e.N) for b in self.keep[6:8]]
        self.big = [pcg.DeviceBuffer(max(8 * e.N, *(8 * n for n in words))) for _ in range(7)]

    def place(self, x_over, z_over):
        """Input buffers 0..4 filled anew; x (z) is the buffer of input x_over
        (z_over), or one of its own (None)."""
        for b, h in zip(self.big, self.host):
            b.upload(h)
        self.x = self.big[5 if x_over is None else x_over]
        self.z = self.big[6 if z_over is None else z_over]
        return [b.ptr for b in self.big[:5]] + [self.x.ptr, self.z.ptr]

    def check(self):
        self.pcg.synchronize()
        assert (self.x.download(np.uint64, self.e.N) == self.want[0]).all()
        assert (self.z.download(np.uint64, self.e.N) == self.want[1]).all()


def expander(pcg, N, c, t):
    e = pcg.Expander(N, c, t, 1, pcg.PRG_CHACHA8, public_a=pcg.public_a(N, c, 7))
    e.set_leaf_shape(64, 8)
    return e


# Inputs 0 roots, 1 correction words, 2 output words, 3 positions, 4 values.
PLACES = [(0, None), (1, None), (2, 3), (None, 3), (None, 4)]


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("N,c,t", [(1 << 14, 2, 8), (1 << 17, 3, 16)])
def test_expand_over_its_inputs(pcg, N, c, t, graph):
    e = expander(pcg, N, c, t)
    r = Request(pcg, e, 11, 1)
    e.set_graph(graph)
    for x_over, z_over in PLACES:
        for _ in range(3):   # with graphs: direct or captured, then replayed
            ptrs = r.place(x_over, z_over)
            e.expand_device(r.party, *ptrs)
            r.check()
    e.close()


def test_expand_batch_over_keys(pcg):
    """x of one request over another's keys."""
    es = [expander(pcg, 1 << 14, 2, 8), expander(pcg, 1 << 14, 4, 16)]
    rs = [Request(pcg, e, 20 + i, i) for i, e in enumerate(es)]
    for over in (0, 1, 2):
        args = [r.place(None, None) for r in rs]
        for r, other, a in zip(rs, rs[::-1], args):
            r.x = other.big[over]
            a[5] = r.x.ptr
        pcg.expand_batch_device([(r.e, r.party, *a) for r, a in zip(rs, args)])
        for r in rs:
            r.check()
    for e in es:
        e.close()


def test_expand_from_g_over_g(pcg):
    N, c, t = 1 << 14, 3, 8
    e = expander(pcg, N, c, t)
    rng = np.random.default_rng(3)
    g = rng.integers(0, pcg.P, c * c * N, dtype=np.uint64)
    pos, val = pcg.noise(N, c, t, 5, 0)
    d_pos, d_val = pcg.to_device(pos), pcg.to_device(val)
    d_g, d_x, d_z = pcg.to_device(g), pcg.DeviceBuffer(8 * N), pcg.DeviceBuffer(8 * N)
    e.expand_from_g_device(d_g.ptr, d_pos.ptr, d_val.ptr, d_x.ptr, d_z.ptr)
    pcg.synchronize()
    want = d_x.download(np.uint64, N), d_z.download(np.uint64, N)
    for block in (0, c * c - 1):
        d_g.upload(g)
        e.expand_from_g_device(d_g.ptr, d_pos.ptr, d_val.ptr, d_g.ptr + 8 * N * block, d_z.ptr)
        pcg.synchronize()
        assert (d_g.download(np.uint64, c * c * N)[N * block:N * (block + 1)] == want[0]).all()
        assert (d_z.download(np.uint64, N) == want[1]).all()
    e.close()


# Walks of one breadth-first stage (n <= 10), of two, and one deeper; the first
# and the last keys' leaves hold the roots.
@pytest.mark.parametrize("prg", ["chacha8", "aes"])
@pytest.mark.parametrize("K,n,w", [(64, 9, 1), (300, 10, 2), (1000, 12, 1), (7, 4, 4)])
def test_keyed_eval_over_its_roots(pcg, K, n, w, prg):
    aes = prg == "aes"
    rng = np.random.default_rng(K + n)
    nk = (1 << w) - 1
    words = lambda k: rng.integers(0, 2**64 - 1, 2 * k, dtype=np.uint64)
    rk = pcg.aes_tree_round_keys(bytes(range(16)), nk) if aes else None
    kind = pcg.PRG_AES if aes else pcg.PRG_CHACHA8
    roots, d_cws = words(K), pcg.to_device(words(K * (n // w) * nk))
    d_roots, d_l = pcg.to_device(roots), pcg.DeviceBuffer(16 * K << n)
    pcg.dpf_keyed_full_eval_device(K, n, w, kind, d_roots.ptr, d_cws.ptr, d_l.ptr, rk)
    pcg.synchronize()
    want = d_l.download(np.uint64, 2 * K << n)
    for at in (0, 16 * ((K << n) - K)):
        d_l.upload_at(roots, at)
        pcg.dpf_keyed_full_eval_device(K, n, w, kind, d_l.ptr + at, d_cws.ptr, d_l.ptr, rk)
        pcg.synchronize()
        assert (d_l.download(np.uint64, 2 * K << n) == want).all()
        # Two groups, each with its roots in the other's leaves.
        d_m = pcg.DeviceBuffer(16 * K << n)
        d_l.upload_at(roots, at)
        d_m.upload_at(roots, at)
        pcg.dpf_keyed_full_eval_multi_device(
            [(K, n, d_m.ptr + at, d_cws.ptr, d_l.ptr), (K, n, d_l.ptr + at, d_cws.ptr, d_m.ptr)],
            w, kind, rk)
        pcg.synchronize()
        assert (d_l.download(np.uint64, 2 * K << n) == want).all()
        assert (d_m.download(np.uint64, 2 * K << n) == want).all()
