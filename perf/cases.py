"""The calls that the speed of this framework is measured on.

Each case is one pass through a public entry point of the package: host and
device inference in the SNICIT and plain modes, one-bit host inputs, uneven
batches in one schedule, one layer alone, and the request server.

Networks come in two kinds.  "generated" ones are drawn by the engine itself
(seeded 32-per-row or RadiX-Net weights, the shapes of the benchmark); "own"
ones are drawn here with numpy and set layer by layer, so that exact() can
evaluate the same network in 64 bits without the package.  Inputs are 0/1 rows
with one density per row (mean 0.19), as the benchmark draws them, except for
the server and the single layers, whose inputs are real numbers.
"""
import numpy as np
import torch

import snicit_gb300 as sg
from snicit_gb300 import serving

BIAS = {256: -0.3, 512: -0.3, 1024: -0.3, 2048: -0.3, 4096: -0.35, 16384: -0.4, 65536: -0.45}
# share of the rows still alive after the first few layers
ALIVE = {256: 0.2, 512: 0.2, 1024: 0.17, 2048: 0.13, 4096: 0.10, 16384: 0.055, 65536: 0.028}
NNZ = 32
VALUE = 0.0625
CLAMP = 32.0
HEAD = 10
_stream = []


def _ptr():
    """The one stream that a program issues its work on."""
    if not _stream:
        _stream.append(torch.cuda.Stream())
    return _stream[0].cuda_stream


def listed():
    return [
        # one small request in the middle of an interactive program: latency and launches only
        {"name": "host-1024x120-b24", "kind": "host", "N": 1024, "L": 120, "rows": 24,
         "mode": "SNICIT", "threshold": 30, "merge": True},
        # an ordinary host batch on a width with no tuned kernel, plain mode
        {"name": "host-2048x60-b600", "kind": "host", "N": 2048, "L": 60, "rows": 600,
         "mode": "SNIG", "threshold": 30, "merge": True},
        # residue rows that last: clustering early, no merging, every post-threshold kernel at work
        {"name": "residue-4096x40-b1500", "kind": "host", "N": 4096, "L": 40, "rows": 1500,
         "mode": "SNICIT", "threshold": 6, "merge": False},
        # the SDGC workloads with the batch resident on the device
        {"name": "sdgc-1024x120-b60000", "kind": "device", "N": 1024, "L": 120, "rows": 60000,
         "mode": "SNICIT", "net": "random"},
        {"name": "sdgc-4096x480-b60000", "kind": "device", "N": 4096, "L": 480, "rows": 60000,
         "mode": "SNICIT", "net": "random"},
        # the plain recurrence on wide rows, an odd row count
        {"name": "plain-16384x48-b6001", "kind": "device", "N": 16384, "L": 48, "rows": 6001,
         "mode": "SNIG", "net": "random"},
        # the widest network (input chunks), fewer layers and rows than the benchmark's 1920 x 60000
        {"name": "sdgc-65536x120-b5000", "kind": "device", "N": 65536, "L": 120, "rows": 5000,
         "mode": "SNICIT", "net": "random"},
        # end to end: float rows in pinned host memory, streamed in while the first layers run
        {"name": "pinned-4096x120-b20000", "kind": "pinned", "N": 4096, "L": 120, "rows": 20000,
         "mode": "SNICIT", "net": "random"},
        # end to end on one-bit rows, on the structured network of the SDGC data
        {"name": "bits-radix-1024x120-b60000", "kind": "bits", "N": 1024, "L": 120, "rows": 60000,
         "mode": "SNICIT", "net": "radixnet"},
        # several users' batches of uneven size in one launch schedule
        {"name": "batches-4096x120-n7", "kind": "batches", "N": 4096, "L": 120, "rows": 9000,
         "count": 7, "mode": "SNICIT", "net": "random"},
        # one hidden layer with a value per edge and a bias per neuron, called from another framework
        {"name": "layer-4096-values-b3001", "kind": "layer", "N": 4096, "rows": 3001,
         "values": True},
        # the request server on the sparse multilayer perceptron with a dense head
        {"name": "serve-1024x24-n48", "kind": "serve", "N": 1024, "L": 24, "rows": 12000,
         "count": 48},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["host", "host", "device", "device", "device", "pinned", "bits", "batches",
                       "layer", "layer", "serve"])
    mode = rng.choice(["SNICIT", "SNICIT", "SNIG"])
    if kind == "host":
        n = rng.choice([256, 512, 1024, 2048, 4096])
        merge = rng.random() < 0.6
        return {"kind": kind, "N": n, "L": _log(rng, 24, min(120, 40 * 4096 // n)),
                "rows": _log(rng, 1, min(2500, 1500 * 4096 // n)), "mode": mode,
                "threshold": rng.choice([6, 12, 20]), "merge": merge}
    if kind == "device":
        n = rng.choice([1024, 4096, 16384, 65536])
        return {"kind": kind, "N": n, "L": _log(rng, 36, min(480, 7000000 // n)),
                "rows": _log(rng, 100, {1024: 60000, 4096: 40000, 16384: 6000, 65536: 2500}[n]),
                "mode": mode, "net": rng.choice(["random", "random", "radixnet"])}
    if kind in ("pinned", "bits"):
        n = rng.choice([1024, 4096])
        return {"kind": kind, "N": n, "L": _log(rng, 36, 120),
                "rows": _log(rng, 1000, {1024: 60000, 4096: 20000}[n]), "mode": mode,
                "net": rng.choice(["random", "radixnet"])}
    if kind == "batches":
        n = rng.choice([1024, 4096])
        return {"kind": kind, "N": n, "L": _log(rng, 36, 120), "rows": _log(rng, 300, 12000),
                "count": rng.randint(2, 12), "mode": "SNICIT", "net": "random"}
    if kind == "layer":
        n = rng.choice([256, 1024, 2048, 4096, 16384])
        return {"kind": kind, "N": n, "rows": _log(rng, 1, min(60000, 3000 * 4096 // n)),
                "values": rng.random() < 0.5}
    return {"kind": kind, "N": 1024, "L": _log(rng, 12, 24), "rows": _log(rng, 500, 12000),
            "count": rng.randint(4, 60)}


# ---- networks and inputs ---------------------------------------------------

def _own_layers(case):
    """(rows, cols, values, bias or None) of each layer, the same for every seed:
    32 out-edges per input, one in each of 32 equal ranges of outputs."""
    n, count = case["N"], case.get("L", 1)
    values = bool(case.get("values"))
    out = []
    for l in range(count):
        g = np.random.default_rng([20260101, n, l, int(values)])
        width = n // NNZ
        c = g.integers(0, width, (n, NNZ), dtype=np.int32) + np.arange(NNZ, dtype=np.int32) * width
        r = np.repeat(np.arange(n, dtype=np.int32), NNZ)
        v = np.full(n * NNZ, VALUE, np.float32)
        b = None
        if values:
            v = (g.standard_normal(n * NNZ) * 0.3).astype(np.float32)
            b = g.uniform(-0.1, 0.0, n).astype(np.float32)
        out.append((r, np.ascontiguousarray(c.reshape(-1)), v, b))
    return out


def _rows01(case, seed, rows=None):
    """0/1 rows on the GPU: density 0.95 * (2nd smallest of 9 uniforms) per row."""
    n, rows = case["N"], case["rows"] if rows is None else rows
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + n)
    rho = 0.95 * torch.rand(rows, 9, generator=g, device="cuda").kthvalue(2, dim=1).values
    y = torch.empty(rows, n, device="cuda")
    step = max(1, (1 << 26) // n)
    for i in range(0, rows, step):
        part = y[i:i + step]
        part.copy_(torch.rand(part.shape, generator=g, device="cuda") < rho[i:i + step, None])
    return y


def _reals(case, seed):
    """Hidden activations of a running network: about a third zero, some at the clamp."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 7)
    y = torch.randn(case["rows"], case["N"], generator=g, device="cuda") * 4 + 2
    return y.clamp_(0.0, CLAMP).contiguous()


def _sizes(case):
    """Sizes of the batches or requests: log-uniform shares of the rows, the same for every seed."""
    g = np.random.default_rng([20260101, case["rows"], case["count"]])
    share = np.exp(g.uniform(0.0, np.log(64.0), case["count"]))
    sizes = np.maximum(1, np.floor(share / share.sum() * case["rows"])).astype(np.int64)
    return [int(s) for s in sizes]


def _engine(case, rows):
    n = case["N"]
    eng = sg.Engine(n, case["L"], mode=case["mode"], threshold=case.get("threshold", 30),
                    batch=rows, bias=BIAS[n], merge=case.get("merge", True))
    if case["kind"] == "host":
        for l, (r, c, v, _) in enumerate(_own_layers(case)):
            eng.set_layer_coo(l, r, c, v)
    elif case["net"] == "radixnet":
        eng.generate_radixnet()
    else:
        eng.generate_weights(20260101)
    eng.finalize()
    return eng


def _pack(y):
    """One bit per entry, entry j in bit j % 64 of 64-bit word j / 64."""
    shift = torch.arange(64, device=y.device, dtype=torch.int64)
    words = []
    for part in y.split(8192):
        b = (part != 0).to(torch.int64).view(part.shape[0], -1, 64)
        words.append((b << shift).sum(2))  # distinct bits: the sum is their union
    return torch.cat(words).cpu().numpy().view(np.uint64)


def prepare(case, seed):
    kind, n = case["kind"], case["N"]
    if kind == "layer":
        eng = sg.Engine(n, 1, mode="SNIG", batch=1, bias=BIAS[n], placement=False)
        (r, c, v, b), = _own_layers(case)
        eng.set_layer_coo(0, r, c, v)
        if b is not None:
            eng.set_layer_bias(0, b)
        eng.finalize()
        y = _reals(case, seed)
        return {"kind": kind, "eng": eng, "y": y, "out": torch.empty_like(y),
                "alive": torch.empty(case["rows"], dtype=torch.int32, device="cuda")}
    if kind == "serve":
        layers, hw, hb = serving.sparse_mlp(20260101, N=n, L=case["L"], H=HEAD)
        eng = sg.Engine(n, case["L"], mode="SNIG", batch=16, bias=-0.05)
        for l, (off, cols, vals) in enumerate(layers):
            eng.set_layer_csr(l, off, cols, vals)
        eng.finalize()
        reqs = [np.random.default_rng([seed, i]).random((s, n), dtype=np.float32)
                for i, s in enumerate(_sizes(case))]
        return {"kind": kind, "reqs": reqs,
                "server": serving.Server(eng, head_w=hw, head_b=hb, slots=3, max_rows=4096)}
    if kind == "batches":
        sizes = _sizes(case)
        eng = _engine(case, sum(sizes))
        y = list(_rows01(case, seed, sum(sizes)).split(sizes))
        flags = [torch.empty(s, dtype=torch.int32, device="cuda") for s in sizes]
        return {"kind": kind, "eng": eng, "y": y, "sizes": sizes, "flags": flags}
    eng = _engine(case, case["rows"])
    y = _rows01(case, seed)
    if kind == "device":
        return {"kind": kind, "eng": eng, "y": y,
                "flags": torch.empty(case["rows"], dtype=torch.int32, device="cuda")}
    if kind == "bits":
        return {"kind": kind, "eng": eng, "y": _pack(y)}
    host = torch.empty(y.shape, pin_memory=kind == "pinned")
    host.copy_(y)
    return {"kind": kind, "eng": eng, "y": host.numpy(), "keep": host}


def run(state):
    kind = state["kind"]
    if kind == "layer":
        y, out, alive = state["y"], state["out"], state["alive"]
        rc = sg.load().sdnn_layer_noalloc(state["eng"]._h, 0, y.data_ptr(), out.data_ptr(),
                                          y.shape[0], alive.data_ptr(), _ptr())
        if rc:
            raise RuntimeError("sdnn_layer_noalloc: status %d" % rc)
        return {"y": out, "alive": alive}
    if kind == "serve":
        server = state["server"]
        got = [server.wait(i) for i in [server.submit(x) for x in state["reqs"]]]
        return {"logits": np.concatenate([g.logits for g in got]),
                "argmax": np.concatenate([g.argmax for g in got]),
                "flags": np.concatenate([g.flags for g in got])}
    eng, y = state["eng"], state["y"]
    if kind == "batches":
        eng.infer_batches_device([x.data_ptr() for x in y], state["sizes"],
                                 [f.data_ptr() for f in state["flags"]], _ptr())
        return state["flags"]
    if kind == "device":
        eng.infer_device(y.data_ptr(), y.shape[0], state["flags"].data_ptr(), _ptr())
        return state["flags"]
    flags, ids = eng.infer_bits(y) if kind == "bits" else eng.infer(y)
    if kind == "host":
        return {"flags": flags, "count": len(ids), "y": eng.activations(y.shape[0])}
    return {"flags": flags, "count": len(ids)}


def work(case):
    """Inputs and weights read once, results written once; the products of the
    rows that are alive (every row in the first two layers; after that the
    plain modes carry the survivors, SNICIT one row per set of equal rows)."""
    kind, n, rows = case["kind"], case["N"], case["rows"]
    if kind == "layer":
        edge = 6 if case["values"] else 2
        return {"bytes": 8.0 * n * rows + 4.0 * rows + float(edge * NNZ * n),
                "flops": 2.0 * NNZ * n * rows}
    if kind == "serve":
        nnz = 0.03 * n * n * case["L"]
        return {"bytes": 4.0 * n * rows + 4.0 * (HEAD + 2) * rows + 6.0 * nnz,
                "flops": 2.0 * nnz * rows + 2.0 * HEAD * n * rows}
    layers = case["L"]
    later = 1.0 if case["mode"] == "SNICIT" and case.get("merge", True) else ALIVE[n] * rows
    read = n / 8.0 if kind == "bits" else 4.0 * n
    back = 4.0 * rows + (4.0 * n * rows if kind == "host" else 0.0)
    return {"bytes": read * rows + back + 2.0 * NNZ * n * layers,
            "flops": 2.0 * NNZ * n * (min(2, layers) * rows + max(0, layers - 2) * max(1.0, later))}


def exact(case, seed):
    kind, n = case["kind"], case["N"]
    if kind == "serve":
        layers, hw, hb = serving.sparse_mlp(20260101, N=n, L=case["L"], H=HEAD)
        y = np.concatenate([np.random.default_rng([seed, i]).random((s, n), dtype=np.float32)
                            for i, s in enumerate(_sizes(case))])
        y = torch.from_numpy(y).double().T.contiguous()
        for off, cols, vals in layers:
            w = torch.sparse_csr_tensor(torch.from_numpy(off.astype(np.int64)),
                                        torch.from_numpy(cols.astype(np.int64)),
                                        torch.from_numpy(vals).double(), (n, n)).to_dense()
            y = (w.T @ y - float(np.float32(0.05))).clamp(0.0, CLAMP)
        return {"logits": (y.T @ torch.from_numpy(hw).double() + torch.from_numpy(hb).double()),
                "argmax": None, "flags": None}
    if kind not in ("host", "layer"):
        return None
    y = (_reals(case, seed) if kind == "layer" else _rows01(case, seed)).cpu().double().T.contiguous()
    for r, c, v, b in _own_layers(case):
        w = torch.sparse_coo_tensor(torch.from_numpy(np.stack([c, r]).astype(np.int64)),
                                    torch.from_numpy(v).double(), (n, n)).to_sparse_csr()
        shift = (float(np.float32(BIAS[n])) if b is None
                 else torch.from_numpy(b).double()[:, None])
        y = (w @ y + shift).clamp_(0.0, CLAMP)
    if kind == "layer":
        return {"y": y.T.contiguous(), "alive": None}
    return {"flags": None, "count": None, "y": y.T.contiguous()}
