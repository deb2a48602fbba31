"""The streamed-list kernel's two ways through a list -- in batches, and as one
stream where a CTA of few rows has its SM to itself -- at the widths and shapes
on both sides of the rule between them.

Both add an output's products in slot order: the rows must agree bit for bit,
and lie within the rounding bound of a sum of n products in FP32,
(n + 2) * 2^-24 * (sum |w y| + |b|), of FP64.
"""
import numpy as np
import pytest

import snicit_gb300 as sg

pytestmark = pytest.mark.gpu


def _net(N, nnz, values, seed):
    rng = np.random.default_rng([seed, N, nnz])
    width = N // nnz
    cols = rng.integers(0, width, (N, nnz)) + np.arange(nnz) * width
    vals = rng.standard_normal(N * nnz) * 0.3 if values else np.full(N * nnz, 0.0625)
    return np.repeat(np.arange(N), nnz), cols.reshape(-1), vals.astype(np.float32)


@pytest.mark.parametrize("values", [False, True])
@pytest.mark.parametrize("N,shapes", [
    (32, [(0, 0), (1, 256), (8, 1024)]), (96, [(0, 0), (2, 512)]), (992, [(0, 0), (4, 1024)]),
    (1024, [(16, 512), (24, 256), (12, 512), (8, 1024)]),
    (4096, [(2, 1024), (3, 512), (4, 512), (5, 512), (6, 512)]),
    (8192, [(0, 0), (2, 512), (1, 256)]),            # 4 rows; 2: two CTAs on an SM
    (16384, [(0, 0), (2, 512), (2, 1024), (1, 512)]),  # stream at 2 x 512 only
    (20480, [(0, 0), (2, 512), (1, 512)]),
    (32768, [(0, 0), (1, 512), (1, 256)]),           # stream with values, and below 1024 threads
])
def test_lists_in_batches_and_as_a_stream_agree(N, shapes, values):
    _same_rows(N, min(32, N // 2), values, shapes, (1, 5, 333))


@pytest.mark.parametrize("values", [False, True])
@pytest.mark.parametrize("N,nnz", [
    (1056, 32), (1088, 32), (1536, 32), (1568, 32), (2080, 32), (2368, 32), (2400, 32), (3072, 32),
    (4064, 32), (1536, 72), (2368, 44), (3072, 72)])  # 72, 44: past the slots that a warp keeps
def test_kept_lists_at_every_stride(N, nnz, values):
    """Widths on both sides of the strides that the kernel with kept lists is
    built for, against lists streamed per tile."""
    _same_rows(N, nnz, values, [(0, 0), (8 if N < 2400 else 4, 512)], (1, 7, 401))


@pytest.mark.parametrize("N,values", [(1056, True), (2080, False)])
def test_many_rows_of_widths_that_fill_the_turns_badly(N, values):
    """Widths where buffers for more than 4096 rows take the other kernel: the
    same bits from an engine with small buffers and from one with large."""
    r, c, v = _net(N, 32, values, 13)
    rng = np.random.default_rng(N)
    Y = np.where(rng.random((4200, N)) < 0.4, rng.random((4200, N)) * 3, 0).astype(np.float32)
    out = []
    for batch in (4096, 4097):
        with sg.Engine(N, 2, mode="SNIG", batch=batch, bias=-0.3) as e:
            for l in range(2):
                e.set_layer_coo(l, r, c, v)
            flags, _ = e.infer(Y[:batch])
            out.append((flags[:4000], e.activations(4000)))
            f, _ = e.infer(Y[:77])
            assert np.array_equal(f, flags[:77])
            assert np.array_equal(e.activations(77).view(np.uint32), out[-1][1][:77].view(np.uint32))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1].view(np.uint32), out[1][1].view(np.uint32))


def _same_rows(N, nnz, values, shapes, counts):
    r, c, v = _net(N, nnz, values, 12)
    bias = -0.2
    rng = np.random.default_rng(N + values)
    order = np.argsort(c, kind="stable")
    n = np.bincount(c, minlength=N)
    start = np.concatenate([[0], np.cumsum(n)])[:-1]
    for rows in counts:
        Y = np.where(rng.random((rows, N)) < 0.4, rng.random((rows, N)) * 3, 0).astype(np.float32)
        got = []
        for tile, threads in shapes:
            with sg.Engine(N, 1, mode="SNIG", batch=rows, bias=bias, tile_rows=tile,
                           threads=threads) as e:
                e.set_layer_coo(0, r, c, v)
                flags, _ = e.infer(Y)
                got.append((flags, e.activations(rows)))
        for flags, act in got[1:]:
            assert np.array_equal(flags, got[0][0])
            assert np.array_equal(act.view(np.uint32), got[0][1].view(np.uint32))
        some = np.unique(np.linspace(0, rows - 1, 12).astype(int))  # FP64: a dozen of the rows
        P = np.zeros((len(some), len(c) + 1))  # (the last column: outputs without edges)
        P[:, :-1] = Y[some][:, r[order]].astype(np.float64) * v[order]
        S, A = (np.where(n > 0, np.add.reduceat(x, start, axis=1), 0) for x in (P, np.abs(P)))
        b = float(np.float32(bias))
        bound = (n + 2) * 2.0 ** -24 * (A + abs(b))
        assert np.all(np.abs(got[0][1][some] - np.clip(S + b, 0, 32)) <= bound)


@pytest.mark.parametrize("N,values", [(1024, False), (1024, True), (1568, True), (3072, False),
                                      (4096, False), (4096, True)])
def test_shares_of_the_sms_change_no_bit(N, values):
    """Passes that take one in 1, 2, 3, 16 or (no CTA left over) 1000 of the SMs,
    few rows and several rounds of tiles, in both modes; launches without rows
    among them."""
    r, c, v = _net(N, 24, values, 14)
    rng = np.random.default_rng(N)
    Y = np.where(rng.random((900, N)) < 0.4, rng.random((900, N)) * 3, 0).astype(np.float32)
    Y[::7] = 0
    for mode in ("SNIG", "SNICIT"):
        with sg.Engine(N, 6, mode=mode, threshold=4, batch=900, bias=-0.1) as e:
            for l in range(6):
                e.set_layer_coo(l, r, c, v)
            for rows in (1, 2, 40, 333, 900):
                want, _ = e.infer(Y[:rows])
                act = e.activations(rows)
                for share in (1, 2, 3, 16, 1000, 0):
                    assert sg.load().sdnn_selftest_share(e._h, share) == 0
                    flags, _ = e.infer(Y[:rows])
                    assert np.array_equal(flags, want), (mode, rows, share)
                    assert np.array_equal(e.activations(rows).view(np.uint32), act.view(np.uint32))


@pytest.mark.parametrize("N,values", [(1024, False), (1024, True), (1568, True), (2400, False),
                                      (4096, False), (4096, True)])
def test_residue_layers_on_either_kernel(N, values):
    """Rows that keep residues to the end (no merging), full and part-filled
    tiles: the kernel with kept lists and the one with lists per tile give the
    same activations, centroids and residue rows."""
    r, c, v = _net(N, 24, values, 15)
    v = np.abs(v)
    v *= np.float32(1.1 / (24 * v.mean()))
    rng = np.random.default_rng(N)
    Y = np.where(rng.random((700, N)) < 0.4, rng.random((700, N)) * 3, 0).astype(np.float32)
    for rows in (40, 700):
        out = []
        for kw in ({}, {"tile_rows": 8 if N < 2400 else 4, "threads": 512}):
            with sg.Engine(N, 5, mode="SNICIT", threshold=2, batch=rows, bias=-0.05, merge=False,
                           sparse_residue=False, num_centroids=4, **kw) as e:
                for l in range(5):
                    e.set_layer_coo(l, r, c, v)
                flags, _ = e.infer(Y[:rows])
                st = e.stats()
                assert st["residue_rows"] > rows // 3 and st["post_kernel"] == 1
                out.append((flags, e.activations(rows), e.layer_rows()))
        for a, b in zip(*out):
            assert np.array_equal(np.ascontiguousarray(a).view(np.uint32),
                                  np.ascontiguousarray(b).view(np.uint32))
