"""The expander's own workspace while its leaf shape changes: the memory stays
where it is large enough, its layout follows the shape of the moment."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Binary AES walks, whose stage plans (and scratch) differ between the shapes:
# from the largest workspace down, and up again.
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("N,c,t", [(1 << 14, 2, 8), (1 << 17, 4, 16)])
def test_leaf_shapes_share_the_workspace(pcg, N, c, t, graph):
    e = pcg.Expander(N, c, t, 1, pcg.PRG_AES, public_a=pcg.public_a(N, c, 7),
                     master_key=np.arange(16, dtype=np.uint8))
    K = e.K
    d_r0, d_r1 = pcg.DeviceBuffer(16 * K), pcg.DeviceBuffer(16 * K)
    d_cws, d_cwo = pcg.DeviceBuffer(16 * K * e.levels), pcg.DeviceBuffer(8 * K)
    e.deal_keys_device(9, d_r0.ptr, d_r1.ptr, d_cws.ptr, d_cwo.ptr)
    noise = [pcg.to_device(v) for v in pcg.noise(N, c, t, 9, 0)]
    d_x, d_z = pcg.DeviceBuffer(8 * N), pcg.DeviceBuffer(8 * N)
    e.set_graph(graph)
    want = None
    for lpt in (4, 8, 16, 8, 4):
        e.set_leaf_shape(32, lpt)
        for _ in range(3):
            pcg.lib.pcgb_memset(d_z.ptr, 0xA5, 8 * N, None)
            e.expand_device(0, d_r0.ptr, d_cws.ptr, d_cwo.ptr, noise[0].ptr, noise[1].ptr,
                            d_x.ptr, d_z.ptr)
            pcg.synchronize()
            got = d_x.download(np.uint64, N), d_z.download(np.uint64, N)
            want = want or got
            assert (got[0] == want[0]).all() and (got[1] == want[1]).all(), lpt
    e.close()
