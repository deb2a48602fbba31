"""The two layer kernels -- slot lists kept in tensor memory (the automatic
choice at N = 1024 .. 4096) and lists streamed per tile (any width; taken when
a tile shape is asked for) -- at the sizes where their splits have edges:
fewer rows than CTAs, a part-filled last tile, widths with a part-filled last
round of groups, and lists deeper than what a warp keeps.

Both add every output's products in the same order, so their rows must agree
bit for bit; and each output must lie within the rounding bound of a sum of
its n products in FP32, (n + 2) * 2^-24 * (sum |w y| + |b|), of FP64.
"""
import numpy as np
import pytest

import snicit_gb300 as sg

pytestmark = pytest.mark.gpu


def _net(N, nnz, values, seed):
    """nnz out-edges per input at distinct outputs; in-degrees vary around nnz."""
    rng = np.random.default_rng([seed, N, nnz])
    width = N // nnz
    cols = rng.integers(0, width, (N, nnz)) + np.arange(nnz) * width
    rows = np.repeat(np.arange(N), nnz)
    vals = rng.standard_normal(N * nnz) * 0.3 if values else np.full(N * nnz, 0.0625)
    return rows, cols.reshape(-1), vals.astype(np.float32)


@pytest.mark.parametrize("N,nnz,values", [
    (1024, 32, False), (1024, 24, True), (1056, 32, False), (2048, 32, True), (2304, 36, False),
    (4096, 32, False), (4096, 20, True),
    (1024, 80, False),   # lists past the 64 slots kept of a group
    (1024, 50, True),    # ... past the 40 kept with their values
    (1024, 200, False),  # too deep to keep: streamed either way
])
def test_resident_and_streamed_lists_agree(N, nnz, values):
    r, c, v = _net(N, nnz, values, 5)
    bias = -0.3
    rng = np.random.default_rng(N + nnz)
    for rows in (1, 7, 153, 1300):
        Y = np.where(rng.random((rows, N)) < 0.4, rng.random((rows, N)) * 3, 0).astype(np.float32)
        Y[rows // 2] = 0  # a row that dies
        got = []
        for kw in ({}, {"tile_rows": 4 if N == 4096 else 8, "threads": 512},
                   {"tile_rows": 2 if N == 4096 else 8, "threads": 1024}):
            with sg.Engine(N, 1, mode="SNIG", batch=rows, bias=bias, **kw) as e:
                e.set_layer_coo(0, r, c, v)
                flags, _ = e.infer(Y)
                got.append((flags, e.activations(rows)))
        for flags, act in got[1:]:
            assert np.array_equal(flags, got[0][0])
            assert np.array_equal(act.view(np.uint32), got[0][1].view(np.uint32))
        W = np.zeros((N, N))
        W[r, c] = v
        Yd, b = Y.astype(np.float64), float(np.float32(bias))
        want = np.clip(Yd @ W + b, 0, 32)
        n = np.bincount(c, minlength=N)
        bound = (n + 2) * 2.0 ** -24 * (Yd @ np.abs(W) + abs(b))
        assert np.all(np.abs(got[0][1] - want) <= bound)
        sure = (Yd @ W + b > bound).any(axis=1) | (Yd @ W + b <= -bound).all(axis=1)
        assert np.array_equal(got[0][0][sure] != 0, (want > 0).any(axis=1)[sure])


@pytest.mark.parametrize("N", [256, 8192, 16384, 32768])
def test_streamed_split_covers_every_row_and_group(N):
    """Row counts around the number of CTAs and of units per tile."""
    r, c, v = _net(N, 32, False, 6)
    bias = -0.3
    rng = np.random.default_rng(N)
    order = np.argsort(c, kind="stable")
    start = np.searchsorted(c[order], np.arange(N + 1))
    for rows in (1, 2, 151, 310):
        Y = np.where(rng.random((rows, N)) < 0.4, rng.random((rows, N)) * 3, 0).astype(np.float32)
        with sg.Engine(N, 1, mode="SNIG", batch=rows, bias=bias) as e:
            e.set_layer_coo(0, r, c, v)
            flags, ids = e.infer(Y)
            act = e.activations(rows)
        P = Y[:, r[order]].astype(np.float64) * 0.0625
        S = np.add.reduceat(P, np.minimum(start[:-1], P.shape[1] - 1), axis=1)
        n = np.diff(start)
        S[:, n == 0] = 0
        b = float(np.float32(bias))
        bound = (n + 2) * 2.0 ** -24 * (S + abs(b))  # inputs and weights >= 0
        assert np.all(np.abs(act - np.clip(S + b, 0, 32)) <= bound)
        assert np.array_equal(np.flatnonzero(flags), ids) and len(ids) == rows


@pytest.mark.parametrize("N,nnz,values,L,K", [
    (1024, 32, False, 70, 1), (1024, 3, False, 35, 3),
    (1024, 80, False, 40, 8),   # lists longer than one batch of 16 blocks
    (1024, 50, True, 36, 2),    # ... than one of 8 with their values
    (4096, 32, False, 67, 1), (4096, 32, False, 10, 4), (4096, 20, True, 36, 1),
    (16384, 20, False, 40, 1),  # one weight buffer
])
def test_chain_carries_the_centroids_like_the_layers(N, nnz, values, L, K):
    """K prototypes, four copies each: after merging, the centroids are all
    there is, and one chain launch over more layers than it looks up at a time
    must give the bits of the per-layer launches."""
    r, c, v = _net(N, nnz, values, 7)
    v = np.abs(v) * np.float32(0.9 / (nnz * np.abs(v).mean()))  # values settle around 1
    rng = np.random.default_rng(N + nnz)
    protos = np.where(rng.random((K, N)) < 0.5, rng.random((K, N)) * 3, 0).astype(np.float32)
    Y = np.tile(protos, (4, 1))
    out = []
    for chain in (True, False):
        with sg.Engine(N, L, mode="SNICIT", threshold=3, batch=4 * K, bias=0.1, num_centroids=50,
                       merge_start=1, chain=chain) as e:
            for l in range(L):
                e.set_layer_coo(l, r, c, v)
            flags, ids = e.infer(Y)
            out.append((flags, e.activations(4 * K), e.stats()))
    st = out[0][2]
    if st["residue_rows"] == 0 and st["centroids"] > 0:
        assert st["post_kernel"] in (2, 3, 4), st
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1].view(np.uint32), out[1][1].view(np.uint32))


@pytest.mark.parametrize("N,nnz,values", [(1024, 32, False), (1056, 32, False), (2048, 32, True),
                                          (4096, 32, False), (4096, 20, True)])
def test_few_rows_share_their_tiles(N, nnz, values):
    """Row counts on both sides of each step of the few-rows split (tiles of 1,
    2, 4 and all rows, then a tile per team): every row must keep the bits that
    it has among many others, whose lists are kept whole."""
    r, c, v = _net(N, nnz, values, 8)
    rng = np.random.default_rng(N)
    all_rows = 2500 if N <= 2048 else 900
    Y = np.where(rng.random((all_rows, N)) < 0.4, rng.random((all_rows, N)) * 3, 0).astype(np.float32)
    Y[3] = 0
    with sg.Engine(N, 2, mode="SNIG", batch=all_rows, bias=-0.3) as e:
        for l in range(2):
            e.set_layer_coo(l, r, c, v)
        flags, _ = e.infer(Y)
        act = e.activations(all_rows)
        for rows in (1, 2, 5, 18, 19, 37, 38, 74, 77, 151, 153, 227, 229, 305, 607, 609):
            if rows > all_rows:
                continue
            f, ids = e.infer(Y[:rows])
            assert np.array_equal(f, flags[:rows]) and np.array_equal(ids, np.flatnonzero(f))
            assert np.array_equal(e.activations(rows).view(np.uint32), act[:rows].view(np.uint32)), rows


@pytest.mark.parametrize("N,rows", [(256, 1), (1024, 31), (1024, 97), (4096, 33), (16384, 40),
                                    (65536, 35)])
@pytest.mark.parametrize("mode", ["SNIG", "SNICIT"])
def test_rows_that_come_as_bits(N, rows, mode):
    """One-bit rows go straight to the counting kernels: same categories and
    activations, bit for bit, as the same rows in floats, in either order of
    calls; ragged last tiles of 32 rows, and fewer rows after more."""
    Y = sg.generate_inputs(N, 11, 0, rows)
    with sg.Engine(N, 3, mode=mode, threshold=2, batch=rows, bias=-0.3) as e:
        e.generate_weights(4)
        for n in (rows, max(1, rows - 7), rows):
            f1, i1 = e.infer(Y[:n])
            a1 = e.activations(n)
            f2, i2 = e.infer_bits(sg.pack_bits(Y[:n]))
            a2 = e.activations(n)
            assert np.array_equal(f1, f2) and np.array_equal(i1, i2)
            assert np.array_equal(a1.view(np.uint32), a2.view(np.uint32))


@pytest.mark.parametrize("N,count,shift", [(256, 1, 0), (1024, 7, 0), (1024, 65, 0), (4096, 5, 0),
                                           (1024, 4, 1)])
def test_device_batches_are_gathered_and_handed_back(N, count, shift):
    """Batches of uneven size, some empty, more than one table of them, and
    inputs that are not aligned to 16 bytes (copied instead): the flags of each
    batch are those of its rows in one batch of all."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(count)
    sizes = [int(s) for s in rng.integers(0, 40, count)]
    sizes[0] = 33
    total = sum(sizes)
    Y = sg.generate_inputs(N, 21, 0, total)
    Y[1::3] = 0
    with sg.Engine(N, 4, mode="SNIG", batch=total, bias=-0.3) as e:
        e.generate_weights(6)
        want, _ = e.infer(Y)
        assert 0 < want.sum() < total
        y, flags, at = [], [], 0
        for s in sizes:
            buf = torch.zeros(max(s, 1) * N + 4, device="cuda")
            part = buf[shift:shift + s * N]
            part.copy_(torch.from_numpy(Y[at:at + s]).reshape(-1))
            y.append((buf, part))
            flags.append(torch.full((max(s, 1),), -7, dtype=torch.int32, device="cuda"))
            at += s
        torch.cuda.synchronize()
        e.infer_batches_device([p.data_ptr() for _, p in y], sizes, [f.data_ptr() for f in flags],
                               torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        at = 0
        for s, f in zip(sizes, flags):
            assert np.array_equal(f.cpu().numpy()[:s], want[at:at + s])
            if s == 0:
                assert int(f[0]) == -7
            at += s


@pytest.mark.parametrize("N,values", [(1024, True), (2048, False), (4096, False), (4096, True)])
def test_passes_that_share_the_sms(N, values):
    """Passes of several slots at once take a share of the SMs each (few rows,
    and a few rounds of tiles): logits and flags of a request are those it gets
    alone, bit for bit."""
    r, c, v = _net(N, 24, values, 9)
    rng = np.random.default_rng(N)
    sizes = [1, 700, 33, 300, 5, 640, 90, 2, 512, 260]
    reqs = [np.where(rng.random((s, N)) < 0.4, rng.random((s, N)) * 3, 0).astype(np.float32)
            for s in sizes]
    hw, hb = rng.standard_normal((N, 4)).astype(np.float32), np.zeros(4, np.float32)
    with sg.Engine(N, 6, mode="SNIG", batch=1024, bias=-0.1) as e:
        for l in range(6):
            e.set_layer_coo(l, r, c, v)
        with sg.Server(e, hw, hb, slots=4, max_rows=1024, max_requests_per_pass=1) as sv:
            alone = [sv.wait(sv.submit(x)) for x in reqs]
            for _ in range(3):
                mix = [sv.wait(i) for i in [sv.submit(x) for x in reqs]]
                for a, m in zip(alone, mix):
                    assert np.array_equal(a.flags, m.flags)
                    assert np.array_equal(a.logits.view(np.uint32), m.logits.view(np.uint32))
