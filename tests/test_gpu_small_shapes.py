"""Expansions whose leaf tiles are shared by clusters of CTAs, and key walks
whose first stage is breadth first, at the sizes where the split changes:
fewest key halves, one tile per bin, ragged keys per CTA, every branching."""
import numpy as np
import pytest

import oracle_lib as O
from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,c,t,w", [(64, 1, 1, 1), (256, 2, 2, 1), (1024, 2, 1, 1),
                                     (1024, 3, 4, 1), (2048, 2, 8, 1), (4096, 2, 32, 2),
                                     (2048, 3, 2, 1), (8192, 2, 16, 2)])
@pytest.mark.parametrize("party", [0, 1])
def test_split_leaf_expansions(pcg, N, c, t, w, party):
    s = O.shape(N, c, t, w)
    r0, r1, cws, cwo = O.deal_keys(s, 77 + N + t)
    a = O.public_a(s, 5)
    roots = (r0, r1)[party]
    pos, val = O.noise(s, 77 + N + t, party)
    want = O.expand(s, party, roots, cws, cwo, pos, val, a)
    e = pcg.Expander(N, c, t, w, pcg.PRG_CHACHA8, public_a=a)
    for tune in (False, True):
        if tune:
            e.autotune()
        x, z = e.expand_host(party, roots, cws, cwo, pos, val)
        assert (x == want[0]).all() and (z == want[1]).all(), (tune, e.leaf_shape())
    e.close()


@pytest.mark.parametrize("prg", [O.PRG_CHACHA8, O.PRG_AES])
@pytest.mark.parametrize("K,n,w", [(1, 1, 1), (3, 9, 1), (5, 10, 1), (2, 11, 1), (1, 4, 4),
                                   (3, 8, 4), (7, 9, 3), (2, 12, 2), (601, 6, 1), (1201, 3, 1)])
def test_breadth_first_walk(pcg, prg, K, n, w):
    nk = (1 << w) - 1
    rng = np.random.default_rng(K * 100 + n)
    roots = rng.integers(0, 2**64 - 1, (K, 2), dtype=np.uint64)
    cws = rng.integers(0, 2**64 - 1, (K * (n // w) * nk, 2), dtype=np.uint64)
    rks = O.aes_tree_round_keys(np.arange(16, dtype=np.uint8), nk) if prg == O.PRG_AES else None
    want = O.dpf_keyed_full_eval(K, n, w, roots, cws, prg, rks).reshape(-1)
    out = pcg.DeviceBuffer(16 * K << n)
    d_r, d_c = dev(pcg, roots), dev(pcg, cws)
    pcg.dpf_keyed_full_eval_device(K, n, w, prg, d_r.ptr, d_c.ptr, out.ptr, round_keys=rks)
    assert (out.download(np.uint64, 2 * (K << n)) == want).all()


@pytest.mark.parametrize("prg", [O.PRG_CHACHA8, O.PRG_AES])
@pytest.mark.parametrize("K,n,w", [(300, 12, 1), (160, 12, 2), (5, 3, 1)])
def test_leaves_at_a_16_byte_address(pcg, prg, K, n, w):
    """A leaf buffer aligned to a node but not to a pair of them."""
    nk = (1 << w) - 1
    rng = np.random.default_rng(K + n)
    roots = rng.integers(0, 2**64 - 1, (K, 2), dtype=np.uint64)
    cws = rng.integers(0, 2**64 - 1, (K * (n // w) * nk, 2), dtype=np.uint64)
    rks = O.aes_tree_round_keys(np.arange(16, dtype=np.uint8), nk) if prg == O.PRG_AES else None
    out = pcg.DeviceBuffer((16 * K << n) + 32)
    d_r, d_c = dev(pcg, roots), dev(pcg, cws)
    words = []
    for off in (0, 16):
        pcg.dpf_keyed_full_eval_device(K, n, w, prg, d_r.ptr, d_c.ptr, out.ptr + off,
                                       round_keys=rks)
        pcg.synchronize()
        words.append(out.download(np.uint64, (2 * K << n) + 2)[off // 8:][:2 * K << n])
    assert (words[0] == words[1]).all()
    few = O.dpf_keyed_full_eval(2, n, w, roots[:2], cws[:2 * (n // w) * nk], prg, rks).reshape(-1)
    assert (words[1][:few.size] == few).all()


# N (the fold's length) on both sides of each step of the shares per output word
# (148 SMs: 18944 and 151552 words), single instances, t = 1, a last row of
# instances cut short, an N beyond the instances' span.
@pytest.mark.parametrize("B,t,D,N", [(1, 1, 2, 1), (1, 1, 64, 100), (1, 4, 32, 64), (3, 4, 32, 70),
                                     (16, 4, 512, 1024), (15, 4, 512, 1031), (49, 7, 1024, 18944),
                                     (64, 8, 4096, 18945), (63, 8, 8192, 32768),
                                     (16, 4, 65536, 151552), (16, 4, 65536, 151553)])
@pytest.mark.parametrize("party", [0, 1])
def test_scatter_with_shared_words(pcg, B, t, D, N, party):
    rng = np.random.default_rng(B * 31 + N)
    leaves = rng.integers(0, 2**64 - 1, (B * D, 2), dtype=np.uint64, endpoint=True)
    leaves[:: 5] = np.uint64(2**64 - 1)
    CW = rng.integers(0, O.P, B, dtype=np.uint64)
    CW[0] = O.P - 1
    want = O.out_scatter_g(leaves, B, D, t, party, CW, N)
    d = dev(pcg, leaves)
    conv, sums = pcg.DeviceBuffer(8 * B * D), pcg.DeviceBuffer(16 * B)
    pcg.dpf_out_convert_device(d.ptr, B, D, conv.ptr, sums.ptr, sums.ptr + 8 * B)
    d_cw, d_g = pcg.to_device(CW), pcg.DeviceBuffer(8 * N)
    for f, src in ((pcg.dpf_out_scatter_g_device, d), (pcg.dpf_out_scatter_g_conv_device, conv)):
        f(src.ptr, B, D, t, party, d_cw.ptr, d_g.ptr, N)
        pcg.synchronize()
        assert (d_g.download(np.uint64, N) == want).all()
