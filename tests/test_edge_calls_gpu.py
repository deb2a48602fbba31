"""Calls at the edges of what the engine takes: infinite clamps, weights that are
loaded anew after a run, buffers that do not fit, in-degrees at the limits of
the counting kernels.
"""
import numpy as np
import pytest

import snicit_gb300 as sg

pytestmark = pytest.mark.gpu


def _identity(N, vals):
    j = np.arange(N)
    return j, j, np.broadcast_to(np.float32(vals), (N,)).copy()


def test_sparse_residues_beside_an_infinite_centroid():
    """With no clamp, a centroid's pre-activation overflows at one neuron.  The
    residue rows equal it there, so their residue stays 0 and they end infinite
    as well (not NaN), as the same rows do without clustering."""
    N, L, rows, hot = 1024, 4, 8, 100
    rng = np.random.default_rng(2)
    Y = np.tile(rng.integers(1, 256, N).astype(np.float32) / 256, (rows, 1))
    Y[:, hot] = 1e30
    for r in range(1, rows):
        Y[r, 7 * r] += 1 / 256  # within the pruning limit of row 0
    up = np.ones(N, np.float32)
    up[hot] = 1e10
    out = []
    for mode in ("SNICIT", "SNIG"):
        with sg.Engine(N, L, mode=mode, threshold=1, batch=rows, bias=0.0, clamp=np.inf,
                       merge=False) as e:
            for l in range(L):
                e.set_layer_coo(l, *_identity(N, up if l == 1 else 1.0))
            flags, _ = e.infer(Y)
            out.append((flags, e.activations(rows)))
            if mode == "SNICIT":
                st = e.stats()
                assert st["centroids"] == 1 and st["sparse_residue_rows"] == rows - 1, st
    want = Y.copy()
    want[:, hot] = np.inf
    for flags, act in out:
        assert flags.all()
        assert np.array_equal(act, want)


def test_stats_of_a_run_whose_weights_were_replaced(tmp_path):
    """Statistics are those of the run, whatever became of its weights: a file
    that loads but is refused when its layers are checked, then good weights
    that take another kernel."""
    torch = pytest.importorskip("torch")
    N, L, rows = 1024, 3, 40
    path = tmp_path / "w.sdnnw"
    with sg.Engine(N, L, mode="SNIG", batch=rows, bias=-0.3) as e:
        e.generate_weights(1)
        e.save_packed(path)
    image = bytearray(path.read_bytes())
    at = 64 + 64 + ((N // 32 + 1) * 4 + 63) // 64 * 64  # the first layer's first slot
    image[at:at + 2] = b"\xff\xff"
    bad = tmp_path / "bad.sdnnw"
    bad.write_bytes(image)
    y = torch.from_numpy(sg.generate_inputs(N, 1, 0, rows)).cuda()
    f = torch.zeros(rows, dtype=torch.int32, device="cuda")
    shape = lambda st: (st["tile_rows"], st["threads"], st["rows_in"])
    with sg.Engine(N, L, mode="SNIG", batch=rows, bias=-0.3) as e:
        e.generate_weights(1)
        e.infer_device(y.data_ptr(), rows, f.data_ptr())
        want = shape(e.stats())
        e.infer_device(y.data_ptr(), rows, f.data_ptr())
        e.load_packed(bad)
        with pytest.raises(sg.SdnnError):
            e.finalize()
        assert shape(e.stats()) == want
        e.generate_weights(1)
        e.infer_device(y.data_ptr(), rows, f.data_ptr())
        e.generate_weights(1, nnz_per_row=200)  # too deep for the kernel of the run
        e.finalize()
        assert shape(e.stats()) == want
        e.infer_device(y.data_ptr(), rows, f.data_ptr())
        assert shape(e.stats()) != want


@pytest.mark.parametrize("values,threads", [(False, 1024), (True, 512)])
def test_stats_name_the_threads_of_the_launch(values, threads):
    """Layers with a value per edge run 512 threads where rows are split into
    input chunks, layers with one value 1024."""
    N, rows = 49152, 3
    j = np.arange(N)
    v = np.full(N, 0.5, np.float32)
    if values:
        v[::2] = 0.25
    with sg.Engine(N, 1, mode="SNIG", batch=rows, bias=0.0) as e:
        e.set_layer_coo(0, j, j[::-1].copy(), v)
        Y = np.random.default_rng(1).integers(0, 8, (rows, N)).astype(np.float32)
        e.infer(Y)
        assert e.stats()["threads"] == threads
        assert np.array_equal(e.activations(rows), (Y * v)[:, ::-1])


@pytest.mark.parametrize("nnz", [-1, 1 << 62])
def test_packed_file_with_a_wrong_edge_count(tmp_path, nnz):
    """The count of edges in a layer's header is for the statistics alone: a
    wrong one changes neither the upload nor the results."""
    N, rows = 1024, 20
    path = tmp_path / "w.sdnnw"
    Y = sg.generate_inputs(N, 1, 0, rows)
    with sg.Engine(N, 2, mode="SNIG", batch=rows, bias=-0.3) as e:
        e.generate_weights(1)
        e.save_packed(path)
        want, _ = e.infer(Y)
    image = bytearray(path.read_bytes())
    image[64 + 8:64 + 16] = nnz.to_bytes(8, "little", signed=True)
    path.write_bytes(image)
    with sg.Engine(N, 2, mode="SNIG", batch=rows, bias=-0.3) as e:
        e.load_packed(path)
        got, _ = e.infer(Y)
    assert 0 < want.sum() < rows and np.array_equal(got, want)


def test_reads_after_buffers_that_did_not_fit():
    """A call whose row buffers cannot be allocated leaves no inference to read
    from; the next one that fits works."""
    torch = pytest.importorskip("torch")
    N, rows = 1024, 8
    Y = sg.generate_inputs(N, 1, 0, rows)
    y = torch.from_numpy(Y).cuda()
    f = torch.zeros(rows, dtype=torch.int32, device="cuda")
    with sg.Engine(N, 2, mode="SNIG", batch=rows, bias=-0.3) as e:
        e.generate_weights(1)
        want, _ = e.infer(Y)
        act = e.activations(rows)
        with pytest.raises(sg.SdnnError) as ei:
            e.infer_device(y.data_ptr(), 1 << 30, f.data_ptr())  # 4 TB a buffer
        assert ei.value.code == 3
        for read in (lambda: e.activations(rows), e.layer_rows):
            with pytest.raises(sg.SdnnError):
                read()
        got, _ = e.infer(Y)
        assert np.array_equal(got, want)
        assert np.array_equal(e.activations(rows).view(np.uint32), act.view(np.uint32))


@pytest.mark.parametrize("N", [992, 1024, 1088, 2400, 4096, 65536])
@pytest.mark.parametrize("mode", ["SNIG", "SNICIT"])
def test_layers_that_no_row_reaches(N, mode):
    """Every row dies in the first layer; the layers after it find none, and the
    next call is as if that one had not been."""
    rows = 70
    Y = sg.generate_inputs(N, 8, 0, rows)
    with sg.Engine(N, 6, mode=mode, threshold=4, batch=rows, bias=-0.01) as e:
        e.generate_weights(3)
        want, _ = e.infer(Y)
        act = e.activations(rows)
        assert want.any()
        for n in (1, rows):
            flags, ids = e.infer(np.zeros((n, N), np.float32))
            assert not flags.any() and len(ids) == 0
            assert not e.activations(n).any()
            assert list(e.layer_rows()) == [n] + [0] * 5
        flags, _ = e.infer(Y)
        assert np.array_equal(flags, want)
        assert np.array_equal(e.activations(rows).view(np.uint32), act.view(np.uint32))


@pytest.mark.parametrize("as_bits", [False, True])
def test_rows_fit_a_full_device_without_the_bit_words(as_bits):
    """A device with room for all of an engine's buffers but the bit words of
    the binary first layer (and, for rows that come as bits, of those): the rows
    run all the same, with the same results."""
    torch = pytest.importorskip("torch")
    N, rows = 16384, 8192
    bits = rows // 32 * N * 4
    Y = np.zeros((rows, N), np.float32)
    Y[:64] = sg.generate_inputs(N, 4, 0, 64)

    def run():
        with sg.Engine(N, 2, mode="SNIG", batch=rows, bias=-0.3, streamed_input=False) as e:
            e.generate_weights(4)
            flags, _ = e.infer(Y)
            act = e.activations(64)
            if not as_bits:
                return flags, act, flags, torch.cuda.mem_get_info()[0]
            f2, _ = e.infer_bits(sg.pack_bits(Y[:70]))
            return flags, act, f2, torch.cuda.mem_get_info()[0]

    torch.zeros(1, device="cuda")
    run()  # (kernels and the context are loaded)
    before = torch.cuda.mem_get_info()[0]
    want = run()
    used = before - want[3]
    leave = used - bits // 2
    filler = []
    for keep in (256 << 20, 0):  # (sizes that the allocator passes on as they are)
        room = torch.cuda.mem_get_info()[0] - leave - keep
        filler.append(torch.empty(room // (2 << 20) * (2 << 20), dtype=torch.uint8, device="cuda"))
    if not leave <= torch.cuda.mem_get_info()[0] < leave + (4 << 20):
        pytest.skip("free device memory cannot be set this closely here")
    got = run()
    del filler
    torch.cuda.empty_cache()
    for a, b in zip(want[:3], got[:3]):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))
    assert want[0].any()


@pytest.mark.parametrize("N", [1024, 4096, 49152])
@pytest.mark.parametrize("degree", [63, 64, 120])
def test_counting_at_the_limits_of_its_planes(N, degree):
    """A binary first layer whose largest in-degree is the last that six planes
    hold, the first that needs seven, and near the most that is counted: rows of
    ones reach that count, and every output is that of the float kernels."""
    rng = np.random.default_rng([N, degree])
    far = np.arange(0, N, 37)  # these outputs have `degree` edges, the others 9
    n = np.full(N, 9)
    n[far] = degree
    cols = np.repeat(np.arange(N), n)
    ins = np.concatenate([rng.permutation(N // 32)[np.arange(k) // 32] * 32 + np.arange(k) % 32
                          for k in n])  # an output's inputs take the banks in turn
    rows = 75
    Y = (rng.random((rows, N)) < np.linspace(0, 1, rows)[:, None]).astype(np.float32)
    Y[-2:] = 1
    got = []
    for counts in (True, False):
        with sg.Engine(N, 1, mode="SNIG", batch=rows, bias=-1.4, binary_first_layer=counts,
                       placement=False) as e:
            e.set_layer_coo(0, ins, cols, np.full(len(ins), 0.0625, np.float32))
            flags, _ = e.infer(Y)
            got.append((flags, e.activations(rows), e.stats()["launches"]))
            if counts:
                f2, _ = e.infer_bits(sg.pack_bits(Y))
                assert np.array_equal(f2, flags)
                assert np.array_equal(e.activations(rows).view(np.uint32), got[0][1].view(np.uint32))
    assert got[0][2] > got[1][2]  # the counting kernels ran
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1].view(np.uint32), got[1][1].view(np.uint32))
    assert got[0][1][-1].max() == np.float32(degree * 0.0625) + np.float32(-1.4)


@pytest.mark.parametrize("N,nnz,values,L,K", [
    (1024, 32, False, 70, 1), (1024, 3, False, 35, 3),
    (1024, 80, False, 40, 8),   # lists longer than one batch of 16 blocks
    (1024, 50, True, 36, 2),    # ... than one of 8 with their values
    (4096, 32, False, 67, 1), (4096, 32, False, 10, 4), (4096, 20, True, 36, 1),
    (16384, 20, False, 40, 1),  # one weight buffer
])
def test_streamed_chain_carries_every_centroid(N, nnz, values, L, K):
    """K prototypes far apart, four copies of each: they are the centroids, no
    residue is left, and the streamed chain runs the layers after the threshold,
    with the bits of a launch per layer and of the chain that reads weights from
    L2."""
    rng = np.random.default_rng([N, nnz, K])
    width = N // nnz
    c = (rng.integers(0, width, (N, nnz)) + np.arange(nnz) * width).reshape(-1)
    r = np.repeat(np.arange(N), nnz)
    v = np.abs(rng.standard_normal(N * nnz)).astype(np.float32) if values else np.ones(N * nnz, np.float32)
    v *= np.float32(0.9 / (nnz * v.mean()))
    protos = np.stack([np.where(rng.random(N) < 0.5, rng.random(N) * 3 * (k + 1), 0)
                       for k in range(K)]).astype(np.float32)
    Y = np.tile(protos, (4, 1))
    out = []
    for kw, kernel in (({}, 3), ({"chain_stream": False}, 2), ({"chain": False}, 1)):
        with sg.Engine(N, L, mode="SNICIT", threshold=3, batch=4 * K, bias=0.1, num_centroids=50,
                       merge_start=1, **kw) as e:
            for l in range(L):
                e.set_layer_coo(l, r, c, v)
            flags, _ = e.infer(Y)
            st = e.stats()
            assert (st["residue_rows"], st["centroids"], st["post_kernel"]) == (0, K, kernel), st
            out.append((flags, e.activations(4 * K)))
    for flags, act in out[1:]:
        assert np.array_equal(flags, out[0][0])
        assert np.array_equal(act.view(np.uint32), out[0][1].view(np.uint32))


@pytest.mark.parametrize("N,rows", [(256, 6200), (1024, 5300), (1056, 300)])
def test_split_of_many_residue_rows(N, rows):
    """Residue rows of 1 to 4 times as many nonzeros as a list holds (and, for the
    larger counts, more rows than the split gives a CTA each): as many become
    lists as must, whichever row is the centroid, and all keep their values."""
    cap = max(32, N // 32)
    rng = np.random.default_rng(N)
    Y = np.tile(rng.integers(1, 200, N).astype(np.float32) / 64, (rows, 1))
    k = rng.integers(0, 4 * cap + 1, rows)  # row r differs from a row s in |k[r] - k[s]| entries
    Y[np.arange(N) < k[:, None]] += np.float32(1 / 256)
    Y = np.ascontiguousarray(Y[:, rng.permutation(N)])
    apart = np.abs(k[:, None] - np.arange(4 * cap + 1))
    expected = list(zip((apart > 0).sum(axis=0), ((apart > 0) & (apart <= cap)).sum(axis=0)))
    out = []
    for sparse in (True, False):
        with sg.Engine(N, 3, mode="SNICIT", threshold=1, batch=rows, bias=0.0, merge=False,
                       num_centroids=1, sparse_residue=sparse) as e:
            for l in range(3):
                e.set_layer_coo(l, *_identity(N, 1.0))
            flags, _ = e.infer(Y)
            st = e.stats()
            out.append((flags, e.activations(rows), list(e.layer_rows())))
            lists = st["sparse_residue_rows"]
            if sparse:
                assert (st["residue_rows"], lists) in expected, (st, k[:5])
                assert 0 < lists < st["residue_rows"] and st["sparse_row_layers"] == 2 * lists
    want = Y
    for flags, act, _ in out:
        assert flags.all()
        assert np.array_equal(act, want)
    assert out[0][2] == out[1][2]
