"""The library from several host threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_stages_of_different_shared_memory(pcg):
    """AES walks whose first stages need 69 and 51 KB of dynamic shared memory:
    one thread's launch does not depend on the other's kernel attributes."""
    rk = pcg.aes_tree_round_keys(bytes(range(16)), 1)
    shapes = [(4736, 12), (64, 10)]
    args, want = [], []
    for i, (K, n) in enumerate(shapes):
        rng = np.random.default_rng(i)
        words = lambda k: rng.integers(0, 2**64 - 1, 2 * k, dtype=np.uint64)
        bufs = pcg.to_device(words(K)), pcg.to_device(words(K * n)), pcg.DeviceBuffer(16 * K << n)
        args.append((K, n, 1, pcg.PRG_AES, *[b.ptr for b in bufs], rk, None, bufs))
    failed, done = [], threading.Event()

    def large():
        try:
            for _ in range(400):
                pcg.dpf_keyed_full_eval_device(*args[0][:-1])
        except Exception as e:
            failed.append(e)
        done.set()

    def small():
        try:
            while not done.is_set():
                pcg.dpf_keyed_full_eval_device(*args[1][:-1])
        except Exception as e:
            failed.append(e)

    for a in args:
        pcg.dpf_keyed_full_eval_device(*a[:-1])
        pcg.synchronize()
        want.append(a[-1][2].download(np.uint64, 2 * a[0] << a[1]))
    th = [threading.Thread(target=f) for f in (large, small)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not failed, failed
    pcg.synchronize()
    for a, w in zip(args, want):
        assert (a[-1][2].download(np.uint64, 2 * a[0] << a[1]) == w).all()


def test_large_host_transfers(pcg):
    """Arrays of 24 MB, moved by helper threads where a call has the staging
    buffer and directly where another call has it; each thread has operands of
    its own (b = X^k), so a crossed buffer shows."""
    N, batch = 1 << 20, 3
    rng = np.random.default_rng(8)
    a = [rng.integers(0, pcg.P, batch * N, dtype=np.uint64) for _ in range(3)]
    ks = [5, 70001, N - 3]
    want, b = [], []
    for v, k in zip(a, ks):
        r = np.roll(v.reshape(batch, N), k, axis=1)
        r[:, :k] = (np.uint64(pcg.P) - r[:, :k]) % np.uint64(pcg.P)
        want.append(r.reshape(-1))
        m = np.zeros((batch, N), np.uint64)
        m[:, k] = 1
        b.append(m.reshape(-1))
    bad = []

    def work(i):
        for _ in range(4):
            got, _ = pcg.poly_mul_u64_gpuntt(a[i], b[i], batch, N)
            if not (got == want[i]).all():
                bad.append(i)

    th = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
