"""Interactive levels with several parents a thread against the oracle, an
instance at a time (instances are independent), leaves and converted words."""
import numpy as np
import pytest

import oracle_lib as O
from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prg", [O.PRG_CHACHA8, O.PRG_AES])
@pytest.mark.parametrize("B,n,w", [(80, 16, 1), (40, 16, 2), (5000, 10, 1)])
def test_large_levels(pcg, B, n, w, prg):
    rng = np.random.default_rng(B + n + w)
    per = (n // w) * ((1 << w) - 1)
    roots = rng.integers(0, 2**64 - 1, (B, 2), dtype=np.uint64)
    dlt = rng.integers(0, 2**64 - 1, (B * per, 2), dtype=np.uint64)
    rks = O.aes_tree_round_keys(np.arange(16, dtype=np.uint8), (1 << w) - 1) if prg == O.PRG_AES else None
    kind = pcg.PRG_AES if prg == O.PRG_AES else pcg.PRG_CHACHA8
    got = pcg.dpf_gpu_batch_full_eval(B, n, w, roots, dlt, rks, prg=kind).reshape(B, -1)
    d_conv, d_s = pcg.DeviceBuffer(8 * B << n), pcg.DeviceBuffer(16 * B)
    pcg.dpf_gpu_batch_full_eval_convert_device(B, n, w, roots, dlt, d_conv.ptr, d_s.ptr,
                                               d_s.ptr + 8 * B, rks, prg=kind)
    conv, sums = d_conv.download(np.uint64, B << n).reshape(B, -1), d_s.download(np.uint64, 2 * B)
    for b in (0, 1, B // 2, B - 1):
        want = O.dpf_batch_full_eval(1, n, w, roots[b:b + 1], dlt[b * per:(b + 1) * per], prg, rks)
        assert (got[b] == want.reshape(-1)).all(), b
        sumC, sumT = O.out_sums(want, 1, 1 << n)
        assert sums[b] == sumC[0] and sums[B + b] == sumT[0], b
        d_l, d_w, d_t = dev(pcg, want), pcg.DeviceBuffer(8 << n), pcg.DeviceBuffer(16)
        pcg.dpf_out_convert_device(d_l.ptr, 1, 1 << n, d_w.ptr, d_t.ptr, d_t.ptr + 8)
        pcg.synchronize()
        assert (conv[b] == d_w.download(np.uint64, 1 << n)).all(), b
