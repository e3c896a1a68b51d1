"""The launch plans of the U-Net's 3x3x3 kernels (csrc/sepx_unet_plan.h, compiled
here) and the walks that the kernels make over them.

Plans: the library's own host code over many layers and volumes -- shared and
tensor memory within an SM's, every output plane and tile once, windows as the
kernels need them, which layers go where.

Walks: numpy restatements of the index arithmetic of conv_zwalk_kernel,
conv_kstream_kernel and conv_wgrad_ring_kernel against direct sums, and their
barriers as actors over mbarriers with parity waits, run in random order: the
TMA or copy warps, the MMA warp, the tensor core that works off its queue, the
epilogue warps.  A slot refilled before its last reader, an accumulator read
before its last term or written before it was read out, a phase that two
completions overtake or a wait that never ends fails."""
import ctypes as C
import random
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
SMEM_SM, RESERVED, SMEM_CTA, COLUMNS = 228 * 1024, 1024, 227 * 1024, 512
LAYERS = [(8, 16), (16, 16), (16, 32), (32, 32), (32, 48), (48, 48), (48, 64), (64, 64), (112, 48), (80, 32), (48, 16)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    so = tmp_path_factory.mktemp("plan") / "plan.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC",
                    f"-I{ROOT / 'sep_code_gb300' / 'csrc'}", str(ROOT / "tests/cpp/unet_plan.cpp"), "-o", str(so)],
                   check=True, capture_output=True, text=True)
    return C.CDLL(str(so))


def _plan(fn, names, *args):
    o = (C.c_longlong * len(names))()
    return dict(zip(names, o)) if fn(*args, o) else None


def zwalk(lib, sms, nb, D, H, W, cin, np_, pool=0):
    return _plan(lib.plan_zwalk, "per_sm nslot ty tx zc nzc nitems grid smem".split(), sms, nb, D, H, W, cin, np_, pool)


def kstream(lib, sms, nb, D, H, W, cin, np_, splits, kper):
    return _plan(lib.plan_kstream, "per_sm nring ty tx zc nzc nitems grid smem nw span".split(), sms, nb, D, H, W, cin,
                 np_, splits, kper)


def ring(lib, sms, nb, D, H, W, cin, cout):
    return _plan(lib.plan_ring, "ncb ngo pw nsy nmb nmbt stacked n ncols na nring njob ty tx zc nzc nitems groups seg "
                 "smem".split(), sms, nb, D, H, W, cin, cout)


def np_of(cout):
    return (cout + 15) // 16 * 16


def split_k(V, cin):
    """conv_any's ranges of a gather or streamed layer: (splits, chunks of one)"""
    kch, mt = (27 * cin + 63) // 64, (V + 127) // 128
    splits, kper = 1, kch
    if mt < 2 * 152 and kch >= 4:
        splits = min((2 * 152 + mt - 1) // mt, kch // 2)
        kper = (kch + splits - 1) // splits
        splits = (kch + kper - 1) // kper
    return splits, kper


def power2(n):
    c = 32
    while c < n:
        c *= 2
    return c


def volumes(seed, n, lo=1, hi=200):
    r = random.Random(seed)
    return [(r.randint(1, 4), *(int(round(np.exp(r.uniform(np.log(lo), np.log(hi))))) for _ in range(3)))
            for _ in range(n)]


# ------------------------------------------------------------------ plans
def test_halo_staged_kernel_keeps_the_wide_layers(lib):
    left = {(cin, n) for cin in range(8, 136, 8) for n in range(16, 144, 16)
            if lib.plan_halo(16, 8, cin, n) and zwalk(lib, 152, 1, 9, 40, 40, cin, n) is None}
    assert left == {(c, n) for c in (8, 16, 24) for n in (96, 112, 128)} | {(32, 96), (32, 112), (40, 80)}
    assert not lib.plan_halo(15, 8, 16, 16) and not lib.plan_halo(16, 7, 16, 16)


@pytest.mark.parametrize("pool", [0, 1])
def test_zwalk_plans(lib, pool):
    for cin, cout in LAYERS + [(8, 1), (24, 24), (40, 48), (32, 80)]:
        n = np_of(cout)
        for nb, D, H, W in volumes(cin + cout, 60) + [(1, 1, 16, 8), (1, 384, 384, 384)]:
            D, H, W = (D, max(H, 16), max(W, 8)) if not pool else (D + D % 2, max(H + H % 2, 16), max(W + W % 2, 8))
            if not lib.plan_halo(H, W, cin, n):
                continue
            p = zwalk(lib, 152, nb, D, H, W, cin, n, pool)
            assert p["smem"] <= SMEM_CTA
            assert p["per_sm"] * ((p["smem"] + 127) // 128 * 128 + RESERVED) <= SMEM_SM
            assert p["per_sm"] * power2(p["zc"] * n) <= COLUMNS and 3 * n <= 256
            assert 1 <= p["zc"] <= 16 and p["nslot"] >= 4
            assert p["zc"] * (p["nzc"] - 1) < D <= p["zc"] * p["nzc"]   # windows cover the planes, none is empty
            assert not pool or p["zc"] % 2 == 0
            assert p["nitems"] == nb * -(-H // 16) * -(-W // 8) * p["nzc"] and 1 <= p["grid"] <= p["nitems"]
    assert zwalk(lib, 152, 1, 4, 16, 8, 16, 16, 1) and zwalk(lib, 152, 1, 5, 16, 8, 16, 16, 1) is None


def test_kstream_plans(lib):
    seen = 0
    for cin, cout in LAYERS + [(128, 128), (208, 16), (160, 16), (16, 128), (48, 112), (24, 16)]:
        n = np_of(cout)
        for nb, D, H, W in volumes(cin * cout, 80) + [(1, 32, 32, 32), (1, 700, 16, 4)]:
            splits, kper = split_k(nb * D * H * W, cin)
            p = kstream(lib, 152, nb, D, H, W, cin, n, splits, kper)
            if p is None:
                continue
            seen += 1
            assert cin % 16 == 0 and p["smem"] <= SMEM_CTA and 2 <= p["nw"] <= 4
            assert p["per_sm"] * ((p["smem"] + 127) // 128 * 128 + RESERVED) <= SMEM_SM
            assert p["per_sm"] * power2(2 * n) <= COLUMNS
            assert 1 <= p["span"] <= 3 and p["span"] <= p["nring"] <= 6
            assert p["zc"] * (p["nzc"] - 1) < D <= p["zc"] * p["nzc"] and (splits == 1 or p["zc"] == 1)
            assert p["nitems"] == nb * -(-H // 16) * -(-W // 8) * p["nzc"] * splits
            for s in range(splits):
                k0, k1 = s * kper * 4, min((s + 1) * kper * 4, 27 * cin // 16)
                assert k0 < k1 and (k1 - 1) // (9 * cin // 16) - k0 // (9 * cin // 16) < p["span"]
    assert seen > 100


def test_ring_plans(lib):
    """also: the default form takes every layer of up to 112 -> 64 channels, so
    that no other form is reached from it"""
    for cin in range(8, 120, 8):
        for cout in (1, 8, 9, 16, 17, 24, 32, 33, 40, 48, 49, 56, 64):
            for nb, D, H, W in volumes(cin * 100 + cout, 12) + [(1, 1, 1, 1), (4, 64, 64, 64)]:
                p = ring(lib, 152, nb, D, H, W, cin, cout)
                assert p is not None and p["smem"] <= SMEM_CTA
                assert p["ncols"] == p["nmb"] * p["nsy"] * (p["n"] if p["stacked"] else 3 * p["n"]) <= COLUMNS
                assert p["n"] <= 256 and p["n"] % 16 == 0 and p["nsy"] in (1, 3) and (p["nsy"] == 1 or p["stacked"])
                assert p["pw"] >= cout and 16 * p["ncb"] >= cin and p["nmb"] in (1, p["nmbt"])
                assert p["njob"] == (3 // p["nsy"]) * (p["nmbt"] // p["nmb"]) and p["njob"] * p["groups"] <= 152
                assert 4 <= p["nring"] <= 12 and 2 <= p["na"] <= 4
                assert p["zc"] * (p["nzc"] - 1) < D <= p["zc"] * p["nzc"]
                assert p["nitems"] == nb * -(-H // 16) * -(-(W + 2) // 8) * p["nzc"] and 1 <= p["groups"] <= p["nitems"]
                assert p["seg"] >= 1
    assert ring(lib, 152, 1, 4, 16, 16, 120, 16) is None and ring(lib, 152, 1, 4, 16, 16, 16, 65) is None


def test_ring_accumulators_take_short_runs(lib):
    """the chains of MMAs that set the weight gradient's error: no longer than
    those of the forms before (tiles of one accumulator)"""
    for layer, vol, most in (((8, 16), (4, 64, 64, 64), 17), ((16, 16), (4, 64, 64, 64), 33), ((32, 48), (4, 64, 64, 64), 47),
                             ((32, 32), (4, 32, 32, 32), 9), ((80, 32), (4, 32, 32, 32), 13),
                             ((112, 48), (2, 64, 64, 64), 80), ((64, 64), (2, 64, 64, 64), 47)):
        assert ring(lib, 152, *vol, *layer)["seg"] <= most, (layer, vol)


# ------------------------------------------------------------------ index arithmetic
def _pad(x):
    return np.pad(x, ((0, 0), (1, 1), (1, 1), (1, 1), (0, 0)))


def _conv(x, w):
    nb, D, H, W, _ = x.shape
    p = _pad(x)
    return sum(p[:, t // 9:t // 9 + D, t // 3 % 3:t // 3 % 3 + H, t % 3:t % 3 + W] @ w[t] for t in range(27))


def _box(x, n, z, y0, x0, rows, cols):
    """rows x columns of plane z from (y0, x0), zeros outside the volume"""
    _, D, H, W, c = x.shape
    out = np.zeros((rows, cols, c))
    if 0 <= z < D:
        ya, yb, xa, xb = max(y0, 0), min(y0 + rows, H), max(x0, 0), min(x0 + cols, W)
        if ya < yb and xa < xb:
            out[ya - y0:yb - y0, xa - x0:xb - x0] = x[n, z, ya:yb, xa:xb]
    return out


def _item(i, p):
    x0, r = i % p["tx"] * 8, i // p["tx"]
    y0, r = r % p["ty"] * 16, r // p["ty"]
    return r // p["nzc"], r % p["nzc"] * p["zc"], y0, x0


@pytest.mark.parametrize("cin,cout,nb,D,H,W,sms", [(16, 16, 2, 7, 17, 9, 3), (8, 16, 1, 1, 16, 8, 2), (48, 32, 1, 20, 18, 11, 2),
                                                   (24, 48, 1, 5, 33, 16, 5)])
def test_zwalk_index_arithmetic(lib, cin, cout, nb, D, H, W, sms):
    p = zwalk(lib, sms, nb, D, H, W, cin, cout)
    rng = np.random.default_rng(cin)
    x, w = rng.standard_normal((nb, D, H, W, cin)), rng.standard_normal((27, cin, cout))
    got = np.full((nb, D, H, W, cout), np.nan)
    for i in range(p["nitems"]):
        n, z0, y0, x0 = _item(i, p)
        nz = min(p["zc"], D - z0)
        d = np.zeros((p["zc"], 128, cout))           # column blocks, from the last output plane to the first
        for j in range((cin + 15) // 16):
            ch = slice(16 * j, min(16 * j + 16, cin))
            for q in range(nz + 2):                  # input plane z0 - 1 + q
                a = _box(x[..., ch], n, z0 - 1 + q, y0 - 1, x0 - 1, 18, 10)
                hi, lo = min(q, nz - 1), max(q - 2, 0)
                for r in range(9):
                    op = a[r // 3:r // 3 + 16, r % 3:r % 3 + 8].reshape(128, -1)
                    for k in range(hi - lo + 1):
                        d[p["zc"] - 1 - hi + k] += op @ w[9 * (q - hi + k) + r][ch]
        for o in range(nz):
            t = d[p["zc"] - 1 - o].reshape(16, 8, cout)
            ny, nx = min(16, H - y0), min(8, W - x0)
            assert np.isnan(got[n, z0 + o, y0:y0 + ny, x0:x0 + nx]).all()
            got[n, z0 + o, y0:y0 + ny, x0:x0 + nx] = t[:ny, :nx]
    assert np.abs(got - _conv(x, w)).max() < 1e-9


@pytest.mark.parametrize("cin,cout,nb,D,H,W,splits,kper", [(112, 48, 1, 5, 17, 16, 1, 48), (112, 48, 1, 3, 32, 24, 3, 16),
                                                           (64, 64, 1, 6, 12, 16, 2, 14), (48, 112, 2, 4, 16, 8, 3, 7)])
def test_kstream_index_arithmetic(lib, cin, cout, nb, D, H, W, splits, kper):
    p = kstream(lib, 4, nb, D, H, W, cin, cout, splits, kper)
    rng = np.random.default_rng(cin)
    x, w = rng.standard_normal((nb, D, H, W, cin)), rng.standard_normal((27, cin, cout))
    c16 = cin // 16
    part = np.full((splits, nb, D, H, W, cout), np.nan)
    for i in range(p["nitems"]):
        s, (n, z0, y0, x0) = i % splits, _item(i // splits, p)
        nz = min(p["zc"], D - z0)
        k0, k1 = s * kper * 4, min((s + 1) * kper * 4, 27 * c16)
        dz0, dz1 = k0 // (9 * c16), (k1 - 1) // (9 * c16)
        planes = [_box(x, n, z0 + dz0 - 1 + q, y0 - 1, x0 - 1, 18, 10) for q in range(nz + dz1 - dz0)]
        for o in range(nz):
            d, kk, tap = np.zeros((128, cout)), k0, k0 // c16
            while kk < k1:
                n16, cg = min((tap + 1) * c16, k1) - kk, kk - tap * c16
                dz, dy, dx = tap // 9, tap // 3 % 3, tap % 3
                op = planes[o + dz - dz0][dy:dy + 16, dx:dx + 8, 16 * cg:16 * (cg + n16)].reshape(128, -1)
                d += op @ w[tap][16 * cg:16 * (cg + n16)]
                kk, tap = kk + n16, tap + 1
            ny, nx = min(16, H - y0), min(8, W - x0)
            assert np.isnan(part[s, n, z0 + o, y0:y0 + ny, x0:x0 + nx]).all()
            part[s, n, z0 + o, y0:y0 + ny, x0:x0 + nx] = d.reshape(16, 8, cout)[:ny, :nx]
    assert np.abs(part.sum(0) - _conv(x, w)).max() < 1e-9


@pytest.mark.parametrize("cin,cout,nb,D,H,W,sms", [(8, 16, 2, 5, 9, 7, 4), (48, 16, 1, 11, 17, 12, 2), (24, 40, 1, 4, 16, 5, 7),
                                                   (48, 48, 1, 6, 16, 16, 9), (112, 56, 1, 3, 7, 6, 12)])
def test_ring_index_arithmetic(lib, cin, cout, nb, D, H, W, sms):
    p = ring(lib, sms, nb, D, H, W, cin, cout)
    rng = np.random.default_rng(cin)
    x, dy = rng.standard_normal((nb, D, H, W, cin)), rng.standard_normal((nb, D, H, W, cout))
    ci, pw = 16 * p["ncb"], p["pw"]
    xp = np.pad(x, ((0, 0),) * 4 + ((0, ci - cin),))
    dp = np.pad(dy, ((0, 0),) * 4 + ((0, pw - cout),))
    dw = np.zeros((27, cin, cout))
    njsy = 3 // p["nsy"]
    for jb in range(p["njob"]):
        sy0, mb0 = jb % njsy * p["nsy"], jb // njsy * p["nmb"]
        for i in range(p["nitems"]):
            n, z0, y0, x0 = _item(i, p)
            for z in range(z0, min(z0 + p["zc"], D)):
                a = _box(dp, n, z, y0, x0 - 2, 16, 10)
                planes = [_box(xp, n, z - 1 + q, y0 - 1, x0 - 1, 18, 8) for q in range(3)]
                for b in range(mb0, mb0 + p["nmb"]):
                    for r in range(64 if pw == 16 or b == 1 else 128):
                        j, m = 2 * b + r // pw, r % pw
                        if j >= 3 or m >= cout:
                            continue
                        row = a[:, j:j + 8, m].reshape(128)             # dY[u - sx], sx = 2 - j
                        for sy in range(sy0, sy0 + p["nsy"]):
                            for dz in range(3):
                                dw[9 * dz + 3 * sy + 2 - j, :, m] += row @ planes[dz][sy:sy + 16].reshape(128, ci)[:, :cin]
    q = _pad(x)
    want = np.stack([np.einsum("nzyxc,nzyxm->cm", q[:, t // 9:t // 9 + D, t // 3 % 3:t // 3 % 3 + H, t % 3:t % 3 + W], dy)
                     for t in range(27)])
    assert np.abs(dw - want).max() < 1e-9


# ------------------------------------------------------------------ barriers
class Bar:
    """an mbarrier: `count` arrivals complete a phase; a wait for a parity passes
    while the phase under way has the other one"""

    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0

    def arrive(self):
        self.left -= 1
        assert self.left >= 0
        if not self.left:
            self.phase, self.left = self.phase + 1, self.count

    def passed(self, parity):
        return self.phase & 1 != parity


class Tensor:
    """MMAs and commits, worked off in order some time after their issue"""

    def __init__(self):
        self.queue = []

    def run(self, over):
        while True:
            yield lambda: self.queue or over()
            if not self.queue:
                return
            self.queue.pop(0)()


def schedule(actors, seed):
    rng = random.Random(seed)
    live = {i: [a, lambda: True] for i, a in enumerate(actors)}
    slow = set(rng.sample(sorted(live), rng.randint(0, 2)))   # laggards: seldom run while others can
    while live:
        ready = [i for i, (_, cond) in live.items() if cond()]
        assert ready, "every actor waits"
        fast = [i for i in ready if i not in slow]
        i = rng.choice(fast if fast and rng.random() < 0.98 else ready)
        # (runs of one actor: the others fall behind)
        for _ in range(rng.choice((1, 1, 3, 20))):
            try:
                live[i][1] = next(live[i][0])
            except StopIteration:
                del live[i]
                break
            if not live[i][1]():
                break


def wait(bar, parity):
    return lambda: bar.passed(parity)


@pytest.mark.parametrize("seed", range(40))
def test_zwalk_barriers(seed):
    rng = random.Random(seed)
    nslot, npair, zc = rng.randint(4, 8), rng.randint(1, 3), rng.randint(1, 7)
    wins = [rng.choice((1, rng.randint(1, zc))) for _ in range(rng.randint(1, 9))]   # planes of this CTA's windows
    zq = (zc + 1) // 2
    full, sfree = [Bar(1) for _ in range(nslot)], [Bar(1) for _ in range(nslot)]
    accf, afree = [Bar(1) for _ in range(zq)], [Bar(4) for _ in range(zq)]
    slots, acc = [None] * nslot, [[] for _ in range(zc)]               # a plane's terms since it was zeroed
    read, issued = [], [False]
    t = Tensor()

    def tma():
        s, ph, filled = 0, 1, 0
        for k, nz in enumerate(wins):
            for j in range(npair):
                for u in range((nz + 3) // 2):
                    if filled == nslot:
                        yield wait(sfree[s], ph)
                    filled = min(filled + 1, nslot)
                    assert slots[s] is None, "slot refilled before its last reader"
                    slots[s] = (k, j, u)
                    full[s].arrive()
                    s, ph = (s + 1) % nslot, ph ^ (s + 1 == nslot)
        yield lambda: True

    def mma():
        s = ph = 0
        for k, nz in enumerate(wins):
            kpar, nu = (k - 1) & 1, (nz + 3) // 2
            for j in range(npair):
                for u in range(nu):
                    yield wait(full[s], ph)
                    if j == 0 and k > 0 and 2 * u < nz:
                        yield wait(afree[u], kpar)

                    def go(s=s, k=k, j=j, u=u, nz=nz):
                        assert slots[s] == (k, j, u)
                        for p in (2 * u, 2 * u + 1):
                            if p < nz + 2:
                                for o in range(max(p - 2, 0), min(p, nz - 1) + 1):
                                    assert not acc[o] or acc[o][-1][0] == k, "added to a plane not read out"
                                    acc[o].append((k, j, p))
                        slots[s] = None
                        sfree[s].arrive()
                    t.queue.append(go)
                    if j == npair - 1 and u >= 1:
                        t.queue.append(accf[u - 1].arrive)
                    s, ph = (s + 1) % nslot, ph ^ (s + 1 == nslot)
            for q in range(nu - 1, zq):
                if k > 0:
                    yield wait(afree[q], kpar)
                t.queue.append(accf[q].arrive)
        issued[0] = True
        yield lambda: True

    state = {}

    def epilogue(half, warp):
        for k, nz in enumerate(wins):
            for q in range(half, zq, 2):
                yield wait(accf[q], k & 1)
                for p in range(2 * q, min(2 * q + 2, nz)):
                    want = [(k, j, i) for j in range(npair) for i in range(p, p + 3)]
                    done = state.setdefault((k, p), [0, list(acc[p])])
                    assert sorted(done[1]) == want, "read before its last term"
                    done[0] += 1
                    if done[0] == 4:
                        acc[p].clear()
                        read.append((k, p))
                yield lambda: True
                afree[q].arrive()
    schedule([tma(), mma(), t.run(lambda: issued[0])] + [epilogue(h, w) for h in (0, 1) for w in range(4)], seed)
    assert sorted(read) == [(k, p) for k, nz in enumerate(wins) for p in range(nz)]


@pytest.mark.parametrize("seed", range(40))
def test_kstream_barriers(seed):
    rng = random.Random(seed)
    span, nw, taps = rng.randint(1, 3), rng.randint(2, 4), rng.randint(1, 4)
    nring = rng.randint(span, 6)
    items = [(rng.randint(1, 4), rng.randint(1, span)) for _ in range(rng.randint(1, 5))]   # output planes, planes of one
    plf, ple = [Bar(8) for _ in range(nring)], [Bar(1) for _ in range(nring)]
    wf, we = [Bar(1) for _ in range(nw)], [Bar(1) for _ in range(nw)]
    accf, afree = [Bar(1) for _ in range(2)], [Bar(4) for _ in range(2)]
    planes, wts, acc = [[] for _ in range(nring)], [None] * nw, [[], []]
    issued, read = [False], []
    t = Tensor()

    def loader(w):
        s, ph, filled, pend = 0, 1, 0, None
        for k, (nz, sp) in enumerate(items):
            for i in range(nz + sp - 1):
                if filled == nring:
                    if not ple[s].passed(ph):
                        if pend is not None:
                            plf[pend].arrive()
                            pend = None
                        yield wait(ple[s], ph)
                filled = min(filled + 1, nring)
                assert all(e[1:] == (k, i) for e in planes[s]), "slot refilled before its last reader"
                planes[s].append((w, k, i))
                yield lambda: True
                if pend is not None:
                    plf[pend].arrive()
                pend = s
                s, ph = (s + 1) % nring, ph ^ (s + 1 == nring)
        if pend is not None:
            plf[pend].arrive()
        yield lambda: True

    def weights():
        s, ph, filled = 0, 1, 0
        for k, (nz, _) in enumerate(items):
            for o in range(nz):
                for tap in range(taps):
                    if filled == nw:
                        yield wait(we[s], ph)
                    filled = min(filled + 1, nw)
                    assert wts[s] is None
                    wts[s] = (k, o, tap)
                    wf[s].arrive()
                    s, ph = (s + 1) % nw, ph ^ (s + 1 == nw)
        yield lambda: True

    def mma():
        ws = wph = ps = pph = os_ = cnt = 0
        for k, (nz, sp) in enumerate(items):
            have = 0
            for o in range(nz):
                b = cnt & 1
                if cnt >= 2:
                    yield wait(afree[b], (cnt >> 1) - 1 & 1)
                for tap in range(taps):
                    dz = min(tap * sp // taps, sp - 1)
                    while have <= o + dz:
                        yield wait(plf[ps], pph)
                        have += 1
                        ps, pph = (ps + 1) % nring, pph ^ (ps + 1 == nring)
                    yield wait(wf[ws], wph)

                    def go(ws=ws, sl=(os_ + dz) % nring, k=k, o=o, tap=tap, i=o + dz, b=b):
                        assert wts[ws] == (k, o, tap) and sorted(planes[sl]) == [(w, k, i) for w in range(8)]
                        assert tap or not acc[b], "accumulator not read out"
                        acc[b].append((k, o, tap))
                        wts[ws] = None
                        we[ws].arrive()
                    t.queue.append(go)
                    ws, wph = (ws + 1) % nw, wph ^ (ws + 1 == nw)
                t.queue.append(accf[b].arrive)
                for _ in range(sp if o == nz - 1 else 1):
                    def release(s=os_):
                        planes[s].clear()
                        ple[s].arrive()
                    t.queue.append(release)
                    os_ = (os_ + 1) % nring
                cnt += 1
        issued[0] = True
        yield lambda: True

    state = {}

    def epilogue(w):
        cnt = 0
        for k, (nz, _) in enumerate(items):
            for o in range(nz):
                b = cnt & 1
                yield wait(accf[b], cnt >> 1 & 1)
                done = state.setdefault((k, o), [0, list(acc[b])])
                assert done[1] == [(k, o, tap) for tap in range(taps)]
                done[0] += 1
                if done[0] == 4:
                    acc[b].clear()
                    read.append((k, o))
                yield lambda: True
                afree[b].arrive()
                cnt += 1
    # (a plane that no tap reads cannot be waited for: every range starts and ends in its first and last plane)
    if taps < span:
        items[:] = [(nz, min(sp, taps)) for nz, sp in items]
    schedule([loader(w) for w in range(8)] + [weights(), mma(), t.run(lambda: issued[0])] + [epilogue(w) for w in range(4)], seed)
    assert sorted(read) == [(k, o) for k, (nz, _) in enumerate(items) for o in range(nz)]


@pytest.mark.parametrize("bias", [0, 1])
@pytest.mark.parametrize("seed", range(40))
def test_ring_barriers(seed, bias):
    rng = random.Random(seed)
    nring, na, seg = rng.randint(4, 12), rng.randint(2, 4), rng.randint(1, 5)
    wins = [rng.randint(1, 6) for _ in range(rng.randint(1, 5))]
    tiles = [(k, z) for k, nz in enumerate(wins) for z in range(nz)]
    plf, ple = [Bar(1) for _ in range(nring)], [Bar(1) for _ in range(nring)]
    af, ae = [Bar(1) for _ in range(na)], [Bar(5 if bias else 1) for _ in range(na)]
    done, drained = Bar(1), Bar(8)
    planes, dys, acc = [None] * nring, [None] * na, [[] for _ in range(8)]   # acc: each epilogue warp's share
    out, summed, issued = [[] for _ in range(8)], [[] for _ in range(4)], [False]
    t = Tensor()

    def loads():
        rs = as_ = pfill = afill = 0
        rph = aph = 1
        for k, nz in enumerate(wins):
            for p in range(nz + 2):
                if pfill == nring:
                    yield wait(ple[rs], rph)
                pfill = min(pfill + 1, nring)
                assert planes[rs] is None, "plane slot refilled before its last reader"
                planes[rs] = (k, p)
                plf[rs].arrive()
                rs, rph = (rs + 1) % nring, rph ^ (rs + 1 == nring)
                if p < 2:
                    continue
                if afill == na:
                    yield wait(ae[as_], aph)
                afill = min(afill + 1, na)
                dys[as_] = (k, p - 2)
                af[as_].arrive()
                as_, aph = (as_ + 1) % na, aph ^ (as_ + 1 == na)
        yield lambda: True

    def mma():
        rs = r0 = as_ = rph = aph = nout = 0
        left = seg
        for k, nz in enumerate(wins):
            for p in range(nz + 2):
                yield wait(plf[rs], rph)
                if p >= 2:
                    yield wait(af[as_], aph)
                rs, rph = (rs + 1) % nring, rph ^ (rs + 1 == nring)
                if p < 2:
                    continue
                r = [(r0 + i) % nring for i in range(3)]

                def go(r=r, a=as_, k=k, p=p):
                    assert [planes[i] for i in r] == [(k, p - 2), (k, p - 1), (k, p)] and dys[a] == (k, p - 2)
                    for share in acc:
                        share.append((k, p - 2))
                t.queue.append(go)
                t.queue.append(ae[as_].arrive)
                for i in r if p == nz + 1 else r[:1]:
                    def release(i=i):
                        planes[i] = None
                        ple[i].arrive()
                    t.queue.append(release)
                r0 = (r[2] + 1) % nring if p == nz + 1 else r[1]
                as_, aph = (as_ + 1) % na, aph ^ (as_ + 1 == na)
                left -= 1
                if left == 0 and not (k == len(wins) - 1 and p == nz + 1):
                    t.queue.append(done.arrive)
                    yield wait(drained, nout & 1)
                    nout, left = nout + 1, seg
        t.queue.append(done.arrive)
        issued[0] = True
        yield wait(done, nout & 1)

    def epilogue(w):
        as_ = aph = 0
        for i, t0 in enumerate(range(0, len(tiles), seg)):
            if bias and w < 4:
                for tile in tiles[t0:t0 + seg]:
                    yield wait(af[as_], aph)
                    assert dys[as_] == tile
                    summed[w].append(tile)
                    yield lambda: True
                    ae[as_].arrive()
                    as_, aph = (as_ + 1) % na, aph ^ (as_ + 1 == na)
            yield wait(done, i & 1)
            assert acc[w] == tiles[t0:t0 + seg], "read out before its last tile, or added to too early"
            out[w] += acc[w]
            acc[w].clear()
            yield lambda: True
            if t0 + seg < len(tiles):
                drained.arrive()
    schedule([loads(), mma(), t.run(lambda: issued[0])] + [epilogue(w) for w in range(8)], seed)
    assert all(o == tiles for o in out) and (not bias or all(s == tiles for s in summed))
