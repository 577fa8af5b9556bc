"""The work this framework is used for, as cases that can be timed one by one.

Every case is one call (or the short run of calls a program makes in a row)
of the package's public entry points on inputs that are already where such a
program has them: keys, noise and polynomials on the device for the
device-pointer entry points, host arrays for the host-buffer ones.  All
outputs are integers (words mod p, check counts), equal bit for bit or wrong.

`work` counts bytes as inputs read once plus outputs written once, and as
"flops" the 32-bit integer operations of the algorithm: 360 per ChaCha8 tree
hash and 341 per output-layer hash (the operations the used output words
need), 320 per AES-128 block (160 table lookups and their XORs), and 20
multiply-add operations per 64-bit modular product of an NTT butterfly or
pointwise pass.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "pcg-square_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import pcg_b200 as L  # noqa: E402

DEV = "cuda:0"
TREE_OPS, OUT_OPS, AES_OPS, MUL_OPS = 360, 341, 320, 20


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # The smallest expansion (N = 2^12, c = 2, t = 4: the two-party
        # bench's shape), repeated on a resident plan with graph replay, as a
        # program that makes many small batches of correlations runs it.
        dict(name="expand_2e12_c2_t4", kind="expand", N=1 << 12, c=2, t=4, w=1, prg="chacha8",
             party=0),
        # A mid-size expansion through the host-buffer API (keys in, x and z
        # out), four-ary tree, three polynomials: one request of a client
        # that keeps its data on the host.
        dict(name="expand_host_2e16_c3_t8_w2", kind="expand_host", N=1 << 16, c=3, t=8, w=2,
             prg="chacha8", party=1),
        # The flagship expansion (N = 2^20, c = 4, t = 16), the largest case.
        dict(name="expand_2e20_c4_t16", kind="expand", N=1 << 20, c=4, t=16, w=1, prg="chacha8",
             party=1),
        # Requests of mixed shapes admitted together, what the server runs for
        # every batch of small requests.
        dict(name="expand_batch_6", kind="expand_batch",
             shapes="14:2:8 16:4:8 14:4:16 18:2:8 16:2:32 15:4:8"),
        # Products of the sizes the v1 poly-mul entry point serves, a few at a
        # time: latency and launches.
        dict(name="polymul_3x2e12", kind="polymul", batch=3, N=1 << 12),
        # The batched-NTT benchmark shape.
        dict(name="polymul_16x2e20", kind="polymul", batch=16, N=1 << 20),
        # Uneven lengths in one call (the mixed-length benchmark, smaller).
        dict(name="polymul_multi_9", kind="polymul_multi", logs="20 16 18 16 20 18 16 17 19"),
        # Keyed full-domain evaluation at the DPF benchmark shape.
        dict(name="dpf_keyed_4096x2e16", kind="dpf_keyed", K=4096, n=16, w=1, prg="chacha8"),
        # The AES tree, an odd number of smaller keys.
        dict(name="dpf_keyed_aes_777x2e14", kind="dpf_keyed", K=777, n=14, w=1, prg="aes"),
        # One block of the reference's device branch through the drop-in
        # entry points: interactive evaluation, output sums, scatter.
        dict(name="dropin_block_2e20_t16", kind="dropin", N=1 << 20, t=16, w=1, prg="chacha8",
             party=0),
        # The online part of a two-party expansion: fused last level, device
        # Beaver multiplication, scatter of the kept words, step 4.
        dict(name="twoparty_2e16_c2_t16", kind="twoparty", N=1 << 16, c=2, t=16, party=1),
        # The consumers: Beaver triples of one party and the OLE check.
        dict(name="triples_verify_2e19", kind="triples", N=1 << 19, party=0),
    ]


def _pow2(rng, lo, hi):
    return 1 << rng.randint(lo, hi)


def draw(rng):
    """One more case of the listed kinds, sizes spread over their logarithm,
    none dearer than the flagship expansion."""
    kind = rng.choice(["expand", "expand", "expand_host", "expand_batch", "polymul", "polymul",
                       "polymul_multi", "dpf_keyed", "dpf_keyed", "dropin", "twoparty", "triples"])
    if kind in ("expand", "expand_host"):
        while True:
            N, c, t = _pow2(rng, 11, 19), rng.randint(2, 4), _pow2(rng, 2, 5)
            prg = rng.choice(["chacha8", "chacha8", "chacha8", "aes"])
            n = int(math.log2(2 * N // t))
            w = rng.choice([1, 1, 2])
            if n % w == 0 and N // t >= 128 and 2 * c * c * t * N <= (1 << 27):
                return dict(kind=kind, N=N, c=c, t=t, w=w, prg=prg, party=rng.randint(0, 1))
    if kind == "expand_batch":
        shapes = []
        for _ in range(rng.randint(2, 9)):
            lg = rng.randint(14, 18)
            shapes.append("%d:%d:%d" % (lg, rng.choice([2, 4]) if lg < 18 else 2,
                                        rng.choice([8, 16, 32])))
        return dict(kind=kind, shapes=" ".join(shapes))
    if kind == "polymul":
        lg = rng.randint(6, 21)
        return dict(kind=kind, batch=rng.randint(1, max(1, min(96, (1 << 24) >> lg))), N=1 << lg)
    if kind == "polymul_multi":
        return dict(kind=kind, logs=" ".join(str(rng.randint(16, 20))
                                             for _ in range(rng.randint(2, 16))))
    if kind == "dpf_keyed":
        n = rng.randint(6, 17)
        K = int(2 ** rng.uniform(2, min(12.5, 26 - n)))
        w = rng.choice([v for v in (1, 1, 2, 3, 4) if n % v == 0])
        return dict(kind=kind, K=K, n=n, w=w, prg=rng.choice(["chacha8", "aes"]))
    if kind == "dropin":
        while True:
            N, t = _pow2(rng, 11, 20), _pow2(rng, 2, 5)
            n, w = int(math.log2(2 * N // t)), rng.choice([1, 1, 2])
            if n % w == 0 and 2 * t * N <= (1 << 25):
                return dict(kind=kind, N=N, t=t, w=w, prg=rng.choice(["chacha8", "chacha8", "aes"]),
                            party=rng.randint(0, 1))
    if kind == "twoparty":
        while True:
            N, c, t = _pow2(rng, 11, 18), rng.randint(2, 4), _pow2(rng, 2, 4)
            if 2 * c * c * t * N <= (1 << 25):
                return dict(kind=kind, N=N, c=c, t=t, party=rng.randint(0, 1))
    return dict(kind="triples", N=_pow2(rng, 9, 21), party=rng.randint(0, 1))


# ---- inputs ------------------------------------------------------------------
class _Rand:
    """Uniform words and residues on the device from a seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed))

    def words(self, n):
        return torch.randint(-(1 << 63), (1 << 63) - 1, (int(n),), dtype=torch.int64, device=DEV,
                             generator=self.g)

    def residues(self, n):
        return torch.randint(0, L.P, (int(n),), dtype=torch.int64, device=DEV, generator=self.g)

    def int(self):
        return int(self.words(1).item()) & ((1 << 62) - 1)


def _host(x):
    return x.cpu().numpy().view(np.uint64)


def _empty(n):
    return torch.empty(int(n), dtype=torch.int64, device=DEV)


def _zeros(n):
    return torch.zeros(int(n), dtype=torch.int64, device=DEV)


def _prg(case):
    return L.PRG_AES if case["prg"] == "aes" else L.PRG_CHACHA8


_MASTER = np.arange(16, dtype=np.uint8)  # AES tree-PRG master key


def _expander(r, N, c, t, w=1, prg=None):
    prg = L.PRG_CHACHA8 if prg is None else prg
    a = _host(r.residues((c - 1) * N))
    return L.Expander(N, c, t, w, prg, public_a=a,
                      master_key=_MASTER if prg == L.PRG_AES else None)


def _dealt(r, e, party):
    """Keys and noise of one request, dealt on the device."""
    r0, r1 = _empty(2 * e.K), _empty(2 * e.K)
    cws, cwo = _empty(2 * e.K * e.levels * e.nk), _empty(e.K)
    seed = r.int()
    torch.cuda.synchronize()
    e.deal_keys_device(seed, r0.data_ptr(), r1.data_ptr(), cws.data_ptr(), cwo.data_ptr())
    pos, val = L.noise(e.N, e.c, e.t, seed, party)
    L.synchronize()
    return dict(roots=r1 if party else r0, cws=cws, cwo=cwo,
                pos=torch.from_numpy(pos.view(np.int64)).to(DEV),
                val=torch.from_numpy(val.view(np.int64)).to(DEV))


def prepare(case, seed):
    r = _Rand(seed)
    kind = case["kind"]
    s = dict(case)
    if kind in ("expand", "expand_host"):
        e = _expander(r, case["N"], case["c"], case["t"], case["w"], _prg(case))
        e.autotune()
        if kind == "expand":
            e.set_graph(True)
        k = _dealt(r, e, case["party"])
        if kind == "expand_host":
            s["host"] = [_host(k[v]) for v in ("roots", "cws", "cwo", "pos", "val")]
        else:
            s.update(x=_empty(e.N), z=_empty(e.N))
        s.update(e=e, k=k)
    elif kind == "expand_batch":
        s["reqs"], s["hold"] = [], []
        for i, sh in enumerate(case["shapes"].split()):
            lg, c, t = (int(v) for v in sh.split(":"))
            e = _expander(r, 1 << lg, c, t)
            e.set_leaf_shape(64, 8)
            k = _dealt(r, e, i & 1)
            x, z = _empty(e.N), _empty(e.N)
            s["hold"].append((e, k, x, z))
            s["reqs"].append((e, i & 1, *(k[v].data_ptr() for v in
                                          ("roots", "cws", "cwo", "pos", "val")),
                              x.data_ptr(), z.data_ptr()))
    elif kind == "polymul":
        n = case["batch"] * case["N"]
        s.update(a=r.residues(n), b=r.residues(n), out=_empty(n))
    elif kind == "polymul_multi":
        lens = [1 << int(v) for v in case["logs"].split()]
        for name, make in (("a", r.residues), ("b", r.residues), ("out", _empty)):
            s[name] = [make(n) for n in lens]
        s["lens"] = lens
    elif kind == "dpf_keyed":
        K, n, w = case["K"], case["n"], case["w"]
        s.update(roots=r.words(2 * K), cws=r.words(2 * K * (n // w) * ((1 << w) - 1)),
                 leaves=_empty(2 * K << n), rk=None)
        if case["prg"] == "aes":
            s["rk"] = L.aes_tree_round_keys(_MASTER, (1 << w) - 1)
    elif kind == "dropin":
        N, t, w = case["N"], case["t"], case["w"]
        B, n = t * t, int(math.log2(2 * N // t))
        s.update(B=B, n=n, roots=_host(r.words(2 * B)),
                 dlt=_host(r.words(2 * B * (n // w) * ((1 << w) - 1))),
                 cw=_host(r.residues(B)), rk=None)
        if case["prg"] == "aes":
            s["rk"] = L.aes_tree_round_keys(_MASTER, (1 << w) - 1)
    elif kind == "twoparty":
        N, c, t = case["N"], case["c"], case["t"]
        e = _expander(r, N, c, t)
        B = e.K
        pos, val = L.noise(N, c, t, r.int(), case["party"])
        s.update(e=e, B=B, n=e.levels, roots=_host(r.words(2 * B)),
                 dlt=_host(r.words(2 * B * e.levels)), beta=r.residues(B), ra=r.residues(B),
                 sa=r.residues(B), rsa=r.residues(B), de_peer=r.residues(2 * B),
                 cw_peer=r.residues(B), de=_empty(2 * B), cw=_empty(B), sumC=_empty(B),
                 sumT=_empty(B), conv=_empty(B << e.levels), g=_empty(c * c * N),
                 pos=torch.from_numpy(pos.view(np.int64)).to(DEV),
                 val=torch.from_numpy(val.view(np.int64)).to(DEV), x=_empty(N), z=_empty(N))
    elif kind == "triples":
        N = case["N"]
        # Two OLEs of both parties that satisfy x0 * x1 = z0 + z1.
        ole = []
        for _ in range(2):
            x0, x1, z0, prod = r.residues(N), r.residues(N), r.residues(N), _empty(N)
            torch.cuda.synchronize()
            L.poly_mul_device(prod.data_ptr(), x0.data_ptr(), x1.data_ptr(), 1, N)
            L.synchronize()
            ole.append((x0, z0, x1, (prod - z0) % L.P))
        s.update(ole=ole, a=_empty(N), b=_empty(N), c=_empty(N), bad=_zeros(2))
    torch.cuda.synchronize()
    return s


# ---- one pass ----------------------------------------------------------------
def _signed(a):
    return a.view(np.int64)


def run(s):
    kind = s["kind"]
    if kind == "expand":
        k = s["k"]
        s["e"].expand_device(s["party"], k["roots"].data_ptr(), k["cws"].data_ptr(),
                             k["cwo"].data_ptr(), k["pos"].data_ptr(), k["val"].data_ptr(),
                             s["x"].data_ptr(), s["z"].data_ptr())
        return s["x"], s["z"]
    if kind == "expand_host":
        x, z = s["e"].expand_host(s["party"], *s["host"])
        return _signed(x), _signed(z)
    if kind == "expand_batch":
        L.expand_batch_device(s["reqs"])
        return [(x, z) for _, _, x, z in s["hold"]]
    if kind == "polymul":
        L.poly_mul_device(s["out"].data_ptr(), s["a"].data_ptr(), s["b"].data_ptr(), s["batch"],
                          s["N"])
        return s["out"]
    if kind == "polymul_multi":
        cnt, vp = len(s["lens"]), L.C.c_void_p
        ptrs = [(vp * cnt)(*[v.data_ptr() for v in s[name]]) for name in ("out", "a", "b")]
        rc = L.lib.pcgb_poly_mul_device_multi(cnt, *ptrs, (L.C.c_int * cnt)(*s["lens"]), None)
        if rc != 0:
            raise RuntimeError(L.lib.pcgb_last_error().decode())
        return s["out"]
    if kind == "dpf_keyed":
        L.dpf_keyed_full_eval_device(s["K"], s["n"], s["w"], _prg(s), s["roots"].data_ptr(),
                                     s["cws"].data_ptr(), s["leaves"].data_ptr(),
                                     round_keys=s["rk"])
        return s["leaves"]
    if kind == "dropin":
        B, n, D = s["B"], s["n"], 1 << s["n"]
        leaves = L.dpf_gpu_batch_full_eval_device(B, n, s["w"], s["roots"], s["dlt"],
                                                  round_keys=s["rk"], party=s["party"],
                                                  prg=_prg(s))
        sumC, sumT = L.dpf_out_sums(leaves, B, D)
        g = L.dpf_out_scatter_g(leaves, B, D, s["t"], s["party"], s["cw"], s["N"])
        return _signed(sumC), _signed(sumT), _signed(g)
    if kind == "twoparty":
        e, B, n, N, c, t, party = (s[v] for v in ("e", "B", "n", "N", "c", "t", "party"))
        D, p = 1 << n, lambda v: s[v].data_ptr()
        L.dpf_gpu_batch_full_eval_convert_device(B, n, 1, s["roots"], s["dlt"], p("conv"),
                                                 p("sumC"), p("sumT"), party=party,
                                                 prg=L.PRG_CHACHA8)
        L.out_beaver_open_device(B, party, p("sumC"), p("sumT"), p("beta"), p("ra"), p("sa"),
                                 p("de"))
        L.out_beaver_close_device(B, party, p("de"), p("de_peer"), p("ra"), p("sa"), p("rsa"),
                                  p("cw"))
        L.add_mod_p_device(p("cw"), p("cw"), p("cw_peer"), B)
        for blk in range(c * c):
            L.dpf_out_scatter_g_conv_device(p("conv") + 8 * blk * t * t * D, t * t, D, t, party,
                                            p("cw") + 8 * blk * t * t, p("g") + 8 * blk * N, N)
        e.expand_from_g_device(p("g"), p("pos"), p("val"), p("x"), p("z"))
        return s["sumC"], s["sumT"], s["cw"], s["g"], s["x"], s["z"]
    (x0, z0, x1, z1), (y0, w0, y1, w1) = s["ole"]
    N, party = s["N"], s["party"]
    mine = (x1, z1, y1, w1) if party else (x0, z0, y0, w0)
    L.triples_device(N, party, *(v.data_ptr() for v in mine), s["a"].data_ptr(),
                     s["b"].data_ptr(), s["c"].data_ptr())
    L.verify_ole_device(N, x0.data_ptr(), z0.data_ptr(), x1.data_ptr(), z1.data_ptr(),
                        s["bad"].data_ptr())
    L.verify_ole_device(N, y0.data_ptr(), w0.data_ptr(), y1.data_ptr(), w1.data_ptr(),
                        s["bad"].data_ptr() + 8)
    return s["a"], s["b"], s["c"], s["bad"]


# ---- what a pass cannot do without --------------------------------------------
def _ntt_ops(N):
    return MUL_OPS * (N // 2) * int(math.log2(N))


def _expand_work(N, c, t, w, prg):
    leaves, K = 2 * c * c * t * N, c * c * t * t
    n = int(math.log2(2 * N // t))
    m = 1 << w
    inner = leaves / (m - 1)                          # internal nodes, each nk hashes
    tree = inner * ((m - 1) * AES_OPS if prg == "aes" else TREE_OPS * math.ceil((m - 1) / 4))
    Q = c * (c + 1) // 2
    ops = tree + leaves * OUT_OPS + (Q + 1) * _ntt_ops(N) + Q * N * MUL_OPS \
        + (c - 1) * t * N * MUL_OPS
    nbytes = K * (16 + 16 * (n // w) * (m - 1) + 8) + 16 * c * t + 8 * (Q + c - 1) * N + 16 * N
    return nbytes, ops


def work(case):
    kind = case["kind"]
    if kind in ("expand", "expand_host"):
        b, f = _expand_work(case["N"], case["c"], case["t"], case["w"], case["prg"])
    elif kind == "expand_batch":
        b = f = 0
        for sh in case["shapes"].split():
            lg, c, t = (int(v) for v in sh.split(":"))
            db, df = _expand_work(1 << lg, c, t, 1, "chacha8")
            b, f = b + db, f + df
    elif kind in ("polymul", "polymul_multi"):
        lens = [case["N"]] * case["batch"] if kind == "polymul" else \
            [1 << int(v) for v in case["logs"].split()]
        b = sum(24 * N for N in lens)
        f = sum(3 * _ntt_ops(N) + MUL_OPS * N for N in lens)
    elif kind == "dpf_keyed":
        K, n, w = case["K"], case["n"], case["w"]
        m = 1 << w
        inner = (K << n) / (m - 1)
        b = (K << n) * 16 + K * 16 * (1 + (n // w) * (m - 1))
        f = inner * ((m - 1) * AES_OPS if case["prg"] == "aes"
                     else TREE_OPS * math.ceil((m - 1) / 4))
    elif kind == "dropin":
        N, t, w = case["N"], case["t"], case["w"]
        B, n, m = t * t, int(math.log2(2 * N // t)), 1 << w
        leaves = 2 * t * N
        b = B * 16 * (1 + (n // w) * (m - 1)) + 24 * B + 8 * N
        f = leaves / (m - 1) * ((m - 1) * AES_OPS if case["prg"] == "aes"
                                else TREE_OPS * math.ceil((m - 1) / 4)) + leaves * OUT_OPS
    elif kind == "twoparty":
        N, c, t = case["N"], case["c"], case["t"]
        b, f = _expand_work(N, c, t, 1, "chacha8")
        b += 8 * c * c * (N + 6 * t * t)
    else:
        N = case["N"]
        b = 8 * N * (4 + 3 + 8)
        f = 9 * _ntt_ops(N) + 3 * N * MUL_OPS
    return {"bytes": float(b), "flops": float(f)}
