"""Host-array entry points on both sides of the copy paths' size limits:
gathered small copies, direct ones, chunks by helper threads (with a ragged
last chunk), outputs over operands, and calls from several threads at once."""
import ctypes as C
import threading

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu
P = O.P


def naive_shift(a, N, k):
    """a * X^k mod X^N + 1 for one polynomial."""
    r = np.roll(a, k)
    r[:k] = (P - r[:k]) % P
    return r


@pytest.mark.parametrize("lg,batch", [(6, 1), (12, 3), (17, 5), (20, 3), (13, 321)])
def test_poly_mul_host_sizes(pcg, lg, batch):
    """b = X^k per polynomial, so the product is a signed rotation of a."""
    N = 1 << lg
    rng = np.random.default_rng(lg)
    a = rng.integers(0, P, batch * N, dtype=np.uint64)
    b = np.zeros((batch, N), np.uint64)
    ks = rng.integers(0, N, batch)
    b[np.arange(batch), ks] = 1
    want = np.concatenate([naive_shift(a[i * N:(i + 1) * N].copy(), N, int(k))
                           for i, k in enumerate(ks)])
    got, _ = pcg.poly_mul_u64_gpuntt(a, b.reshape(-1), batch, N)
    assert (got == want).all()
    out = a.copy()   # output over the first operand
    rc = pcg.lib.pcgb_poly_mul_u64(pcg.POLYMUL_MERGE, out, out, b.reshape(-1).copy(), batch, N, P,
                                   C.byref(C.c_double()))
    assert rc == 0 and (out == want).all()
    pcg.trim_pool()   # the staging buffer comes back on the next call


def test_host_calls_from_threads(pcg):
    N = 1 << 15
    rng = np.random.default_rng(5)
    a = rng.integers(0, P, 4 * N, dtype=np.uint64)
    b = rng.integers(0, P, 4 * N, dtype=np.uint64)
    want, _ = pcg.poly_mul_u64_gpuntt(a, b, 4, N)
    bad = []

    def work():
        for _ in range(5):
            got, _ = pcg.poly_mul_u64_gpuntt(a, b, 4, N)
            if not (got == want).all():
                bad.append(1)

    th = [threading.Thread(target=work) for _ in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad


def test_interactive_levels_without_exchange(pcg):
    """No callback means zero peer shares on every level, as a callback that
    returns zeros; large levels (several parents a thread) included."""
    for B, n, w in ((3, 6, 1), (5, 4, 2), (80, 16, 1), (40, 16, 2)):
        rng = np.random.default_rng(n + w)
        roots = rng.integers(0, 2**64 - 1, (B, 2), dtype=np.uint64)
        dlt = rng.integers(0, 2**64 - 1, (B * (n // w) * ((1 << w) - 1), 2), dtype=np.uint64)
        none = pcg.dpf_gpu_batch_full_eval(B, n, w, roots, dlt, prg=pcg.PRG_CHACHA8)
        zero = pcg.dpf_gpu_batch_full_eval(B, n, w, roots, dlt, prg=pcg.PRG_CHACHA8,
                                           exchange=lambda m: np.zeros_like(m))
        assert (none == zero).all()
        d_conv, d_s = pcg.DeviceBuffer(8 * B << n), pcg.DeviceBuffer(16 * B)
        pcg.dpf_gpu_batch_full_eval_convert_device(B, n, w, roots, dlt, d_conv.ptr, d_s.ptr,
                                                   d_s.ptr + 8 * B, prg=pcg.PRG_CHACHA8)
        conv = d_conv.download(np.uint64, B << n)
        assert ((conv >> np.uint64(63)) == (none[:, 0] & np.uint64(1))).all()
        ref = pcg.DeviceBuffer(16 * B)
        d_l = pcg.to_device(none)
        d_c2 = pcg.DeviceBuffer(8 * B << n)
        pcg.dpf_out_convert_device(d_l.ptr, B, 1 << n, d_c2.ptr, ref.ptr, ref.ptr + 8 * B)
        pcg.synchronize()
        assert (d_c2.download(np.uint64, B << n) == conv).all()
        assert (ref.download(np.uint64, 2 * B) == d_s.download(np.uint64, 2 * B)).all()


@pytest.mark.parametrize("t,D,N", [(4, 1 << 17, 1 << 18), (8, 1 << 17, 1 << 19),
                                   (5, 1 << 17, 700001), (4, 1 << 18, 6000000)])
def test_scatter_in_pieces(pcg, t, D, N):
    """g copied out piece by piece equals the device form's, past the fold and
    in the zero tail of an N larger than the instances span."""
    B = t * t
    leaves = pcg.DeviceBuffer(16 * B * D)
    rng = np.random.default_rng(t)
    block = rng.integers(0, 2**64 - 1, 2 * D, dtype=np.uint64)
    for b in range(B):
        leaves.upload_at(np.roll(block, 2 * b), 16 * b * D)
    CW = rng.integers(0, 2**64 - 1, B, dtype=np.uint64)
    d_cw, d_g = pcg.to_device(CW % np.uint64(P)), pcg.DeviceBuffer(8 * N)
    for party in (0, 1):
        g = pcg.dpf_out_scatter_g(leaves.ptr, B, D, t, party, CW, N)
        pcg.dpf_out_scatter_g_device(leaves.ptr, B, D, t, party, d_cw.ptr, d_g.ptr, N)
        pcg.synchronize()
        assert (g == d_g.download(np.uint64, N)).all()
