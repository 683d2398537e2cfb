"""Workloads of the skeleton runtime for timing and for comparing two builds.

Each case is a call sequence a user's program makes through
`skelcl_gb300.Program.launch` (and the C ABI's adjoint entry points): the
skeletons are constructed once per process, as a SkelCL program does, the
buffers belong to the caller and every pass is given the same kind of data a
first pass gets.  Forward and adjoint run on the library's stream; nothing
waits for the device inside `run`.
"""
import math

import numpy as np
import torch

import skelcl_gb300 as S

# element types: name -> (OpenCL C spelling, torch, numpy)
TYPES = {
    "float": ("float", torch.float32, np.float32),
    "double": ("double", torch.float64, np.float64),
    "int": ("int", torch.int32, np.int32),
    "uchar": ("unsigned char", torch.uint8, np.uint8),
}
MOD = 7919


def listed():
    return [
        # the smallest calls: a dot product of a short vector, two launches,
        # where what counts is the latency of a call
        {"name": "dot_1e3", "kind": "dot", "n": 1000, "dtype": "float"},
        # the dot product example at its default length (2^24)
        {"name": "dot_2e24", "kind": "dot", "n": 1 << 24, "dtype": "float"},
        # inclusive integer prefix sum, then a Map over it: the headline
        # workload of the benchmark, HBM-sized
        {"name": "scan_mod_2e28", "kind": "scan_mod", "n": 1 << 28},
        # a differentiated float prefix sum: forward and reverse scan
        {"name": "scan_train_2e26", "kind": "scan_train", "n": 1 << 26, "dtype": "float", "inclusive": True},
        # a differentiated element-wise Map of an odd length
        {"name": "map_train_5e7", "kind": "map_train", "n": 50_000_003, "dtype": "float"},
        # Gaussian blur of a large image and its gradient (11 x 11 taps,
        # clamped borders): the benchmark's stencil
        {"name": "blur_train_8192_r5", "kind": "blur_train", "rows": 8192, "cols": 8192, "r": 5, "nearest": True},
        # an edge filter over an 8-bit camera frame: a small stencil, bytes
        {"name": "sobel_u8_1080p", "kind": "sobel", "rows": 1080, "cols": 1920},
        # matrix multiplication as AllPairs, the benchmark's size
        {"name": "matmul_8192_4096", "kind": "matmul", "m": 8192, "k": 4096, "n": 8192},
        # a dense layer of ordinary, ragged size: forward, both gradients
        {"name": "matmul_train_1000", "kind": "matmul_train", "m": 1000, "k": 500, "n": 1100},
        # Manhattan distances of two point sets: AllPairs on the CUDA cores
        {"name": "distance_4096_256", "kind": "distance", "m": 4096, "k": 256, "n": 4096},
        # 10,000 vectors of very uneven length back to back: Map, Scan,
        # Reduce per vector and their adjoints (the benchmark's batch)
        {"name": "segments_train_1e4", "kind": "segments_train", "vectors": 10_000, "law": "log", "lo": 64,
         "hi": 1 << 20},
        # a million short vectors, as ragged batches of records have them
        {"name": "segments_train_1e6", "kind": "segments_train", "vectors": 1_000_000, "law": "even", "lo": 1,
         "hi": 200},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dot", "scan_mod", "scan_train", "map_train", "blur_train", "sobel", "matmul",
                       "matmul_train", "distance", "segments_train", "segments_short"])
    if kind == "dot":
        return {"kind": kind, "n": _log(rng, 200, 1 << 25), "dtype": rng.choice(["float", "double", "int"])}
    if kind == "scan_mod":
        return {"kind": kind, "n": _log(rng, 500, (1 << 28) - 1)}
    if kind == "scan_train":
        return {"kind": kind, "n": _log(rng, 500, (1 << 26) - 1), "dtype": rng.choice(["float", "double"]),
                "inclusive": rng.random() < 0.5}
    if kind == "map_train":
        return {"kind": kind, "n": _log(rng, 500, 1 << 26), "dtype": rng.choice(["float", "double"])}
    if kind == "blur_train":
        return {"kind": kind, "rows": _log(rng, 60, 8191), "cols": _log(rng, 60, 8191),
                "r": rng.choice([1, 2, 3, 5]), "nearest": rng.random() < 0.5}
    if kind == "sobel":
        return {"kind": kind, "rows": _log(rng, 60, 8000), "cols": _log(rng, 60, 8000)}
    if kind == "matmul":
        return {"kind": kind, "m": _log(rng, 64, 8000), "k": _log(rng, 16, 4000), "n": _log(rng, 64, 8000)}
    if kind == "matmul_train":
        return {"kind": kind, "m": _log(rng, 64, 4000), "k": _log(rng, 64, 4000), "n": _log(rng, 64, 4000)}
    if kind == "distance":
        return {"kind": kind, "m": _log(rng, 64, 4090), "k": _log(rng, 8, 256), "n": _log(rng, 64, 4090)}
    if kind == "segments_train":
        return {"kind": kind, "vectors": _log(rng, 50, 9000), "law": "log", "lo": rng.choice([1, 16, 64]),
                "hi": _log(rng, 1 << 12, 1 << 20)}
    return {"kind": "segments_train", "vectors": _log(rng, 2000, 900_000), "law": "even",
            "lo": rng.choice([0, 1]), "hi": _log(rng, 8, 400)}


# ---- skeletons, constructed once per process --------------------------------------
_built = {}

ADD = "{t} func({t} x, {t} y){{ return x + y; }}"
MUL = "{t} func({t} x, {t} y){{ return x * y; }}"


def _program(key, kind, source, types, **kw):
    if key not in _built:
        S.init(0)
        _built[key] = S.Program(kind, source, types, **kw)
    return _built[key]


def _add(kind, dtype):
    t = TYPES[dtype][0]
    return _program((kind, dtype), kind, ADD.format(t=t), [t], identity="0")


def _mul(dtype):
    t = TYPES[dtype][0]
    return _program(("mul", dtype), S.KIND_ZIP, MUL.format(t=t), [t] * 3)


def _square(dtype):
    t = TYPES[dtype][0]
    return _program(("square", dtype), S.KIND_MAP, f"{t} func({t} x){{ return x * x + 1; }}", [t, t])


def _square_adjoint(dtype):
    t = TYPES[dtype][0]
    return _program(("square_adjoint", dtype), S.KIND_MAP_ADJOINT, f"{t} d({t} x, {t} g){{ return 2 * x * g; }}",
                    [t, t], func="d")


def _stencil(r, padding):
    w = 2 * r + 1
    src = ("float func(input_matrix_t img, __global float* w) { float s = 0.0f;"
           f" for (int dy = -{r}; dy <= {r}; ++dy) for (int dx = -{r}; dx <= {r}; ++dx)"
           f"  s += getData(img, dx, dy) * w[(dy + {r}) * {w} + (dx + {r})]; return s; }}")
    return _program(("stencil", r, padding), S.KIND_MAPOVERLAP, src, ["float", "float"], overlap_range=r,
                    padding=padding, neutral="0.0f")


SOBEL = ("unsigned char func(input_matrix_t img) {"
         " int gx = getData(img, 1, -1) + 2 * getData(img, 1, 0) + getData(img, 1, 1)"
         "  - getData(img, -1, -1) - 2 * getData(img, -1, 0) - getData(img, -1, 1);"
         " int gy = getData(img, -1, 1) + 2 * getData(img, 0, 1) + getData(img, 1, 1)"
         "  - getData(img, -1, -1) - 2 * getData(img, 0, -1) - getData(img, 1, -1);"
         " int s = (gx < 0 ? -gx : gx) + (gy < 0 ? -gy : gy); return s > 255 ? 255 : s; }")


def _pairs(zip_expr):
    return _program(("pairs", zip_expr), S.KIND_ALLPAIRS, ADD.format(t="float"), ["float"] * 3,
                    source2=f"float func(float x, float y){{ return {zip_expr}; }}", identity="0")


# ---- inputs ------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, dtype, lo=-1.0, hi=1.0):
    t = TYPES[dtype][1]
    if dtype == "int":
        return torch.randint(-1000, 1001, (n,), generator=g, device="cuda", dtype=t)
    return torch.rand(n, generator=g, device="cuda", dtype=t) * (hi - lo) + lo


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _weights(r):
    """Normalised Gaussian weights of radius r (float32, row-major)."""
    s = max(r / 2.5, 0.5)
    y, x = np.mgrid[-r:r + 1, -r:r + 1]
    w = np.exp(-(x * x + y * y) / (2.0 * s * s))
    return (w / w.sum()).astype(np.float32)


def _lengths(case, seed):
    """The vectors' lengths: the same ones for a case, in an order of the seed's."""
    rng = np.random.default_rng(case["vectors"])
    if case["law"] == "log":
        e = rng.uniform(math.log2(case["lo"]), math.log2(case["hi"]), case["vectors"])
        lens = np.floor(2.0 ** e).astype(np.int64)
    else:
        lens = rng.integers(case["lo"], case["hi"], case["vectors"])
    return np.random.default_rng(int(seed)).permutation(lens)


def _inputs(case, seed):
    """The case's inputs: CUDA tensors (and host arrays for weights)."""
    g, kind = _gen(seed), case["kind"]
    if kind == "dot":
        return {"x": _uniform(g, case["n"], case["dtype"]), "y": _uniform(g, case["n"], case["dtype"])}
    if kind == "scan_mod":
        return {"x": torch.randint(0, 1001, (case["n"],), generator=g, device="cuda", dtype=torch.int32)}
    if kind in ("scan_train", "map_train"):
        return {"x": _uniform(g, case["n"], case["dtype"]), "g": _uniform(g, case["n"], case["dtype"])}
    if kind == "blur_train":
        n = case["rows"] * case["cols"]
        return {"x": _uniform(g, n, "float", 0.0, 255.0), "g": _uniform(g, n, "float"), "w": _weights(case["r"])}
    if kind == "sobel":
        return {"x": torch.randint(0, 256, (case["rows"] * case["cols"],), generator=g, device="cuda",
                                   dtype=torch.uint8)}
    if kind in ("matmul", "matmul_train", "distance"):
        m, k, n = case["m"], case["k"], case["n"]
        d = {"a": _normal(g, m, k), "b": _normal(g, k, n)}
        if kind == "matmul_train":
            d["g"] = _normal(g, m, n)
        return d
    lens = _lengths(case, seed)
    off = np.concatenate([[0], np.cumsum(lens)])
    n = int(off[-1])
    return {"x": _uniform(g, n, "float"), "g": _uniform(g, len(lens), "float"), "n": n,
            "off": torch.from_numpy(off).to("cuda")}


def _dev(t):
    """The library's view of a caller's CUDA tensor."""
    names = {torch.float32: np.float32, torch.float64: np.float64, torch.int32: np.int32, torch.uint8: np.uint8,
             torch.int64: np.uint64}
    return S.DeviceArray(t.numel(), names[t.dtype], ptr=t.data_ptr())


def prepare(case, seed):
    S.init(0)
    i, kind = _inputs(case, seed), case["kind"]
    st = {"case": case, "kind": kind}
    if kind == "dot":
        d = case["dtype"]
        st["mul"], st["sum"] = _mul(d), _add(S.KIND_REDUCE, d)
        i["z"], i["r"] = torch.empty_like(i["x"]), torch.empty(1, device="cuda", dtype=i["x"].dtype)
    elif kind == "scan_mod":
        st["scan"] = _add(S.KIND_SCAN, "int")
        st["mod"] = _program("mod", S.KIND_MAP, "int func(int x){ return x % %d; }".replace("%d", str(MOD)),
                             ["int", "int"])
        i["s"], i["o"] = torch.empty_like(i["x"]), torch.empty_like(i["x"])
    elif kind == "scan_train":
        st["scan"] = _add(S.KIND_SCAN, case["dtype"])
        i["s"], i["gx"] = torch.empty_like(i["x"]), torch.empty_like(i["x"])
    elif kind == "map_train":
        st["map"], st["adj"] = _square(case["dtype"]), _square_adjoint(case["dtype"])
        i["m"], i["gx"] = torch.empty_like(i["x"]), torch.empty_like(i["x"])
    elif kind == "blur_train":
        w = i["w"]
        i["w"] = torch.from_numpy(w.ravel()).to("cuda")
        i["wt"] = torch.from_numpy(np.ascontiguousarray(w[::-1, ::-1]).ravel()).to("cuda")
        st["blur"] = _stencil(case["r"], S.PAD_NEAREST if case["nearest"] else S.PAD_NEUTRAL)
        st["adj"] = _stencil(case["r"], S.PAD_NEUTRAL)
        i["o"], i["gx"] = torch.empty_like(i["x"]), torch.empty_like(i["x"])
    elif kind == "sobel":
        st["filter"] = _program("sobel", S.KIND_MAPOVERLAP, SOBEL, ["unsigned char"] * 2, overlap_range=1,
                                padding=S.PAD_NEAREST)
        i["o"] = torch.empty_like(i["x"])
    elif kind in ("matmul", "matmul_train", "distance"):
        st["pairs"] = _pairs("fabs(x - y)" if kind == "distance" else "x * y")
        i["p"] = torch.empty(case["m"], case["n"], device="cuda")
        if kind == "matmul_train":
            i["ga"], i["gb"] = torch.empty_like(i["a"]), torch.empty_like(i["b"])
    else:
        st["map"], st["madj"] = _square("float"), _square_adjoint("float")
        st["scan"], st["sum"] = _add(S.KIND_SCAN, "float"), _add(S.KIND_REDUCE, "float")
        for k in ("m", "s", "gs", "gm", "gx"):
            i[k] = torch.empty_like(i["x"])
        i["r"] = torch.empty_like(i["g"])
        st["n"] = i.pop("n")
    st["t"] = i
    st["d"] = {k: _dev(t) for k, t in i.items()}
    torch.cuda.synchronize()  # the inputs were made on torch's stream
    if kind == "segments_train":
        st["plan"] = S.SegPlan(st["d"]["off"], st["n"])
    return st


def run(st):
    kind, case, t, d = st["kind"], st["case"], st["t"], st["d"]
    if kind == "dot":
        st["mul"].launch([d["x"], d["y"], d["z"]], n=case["n"])
        st["sum"].launch([d["z"], d["r"]], n=case["n"])
        return [t["z"], t["r"]]
    if kind == "scan_mod":
        st["scan"].launch([d["x"], d["s"]], n=case["n"], flags=S.SHAPE_INCLUSIVE)
        st["mod"].launch([d["s"], d["o"]], n=case["n"])
        return [t["s"], t["o"]]
    if kind == "scan_train":
        f = S.SHAPE_INCLUSIVE if case["inclusive"] else 0
        st["scan"].launch([d["x"], d["s"]], n=case["n"], flags=f)
        st["scan"].launch([d["g"], d["gx"]], n=case["n"], flags=f | S.SHAPE_REVERSE)
        return [t["s"], t["gx"]]
    if kind == "map_train":
        st["map"].launch([d["x"], d["m"]], n=case["n"])
        st["adj"].launch([d["x"], d["g"], d["gx"]], n=case["n"])
        return [t["m"], t["gx"]]
    if kind == "blur_train":
        rows, cols = case["rows"], case["cols"]
        st["blur"].launch([d["x"], d["o"]], rows=rows, cols=cols, extra=S.buffer(d["w"]))
        st["adj"].launch([d["g"], d["gx"]], rows=rows, cols=cols, extra=S.buffer(d["wt"]))
        if case["nearest"]:
            S.check(S.lib().scl_mapoverlap_adjoint_edges(d["g"].ptr, d["wt"].ptr, d["gx"].ptr, rows, cols, case["r"]))
        return [t["o"], t["gx"]]
    if kind == "sobel":
        st["filter"].launch([d["x"], d["o"]], rows=case["rows"], cols=case["cols"])
        return [t["o"]]
    if kind in ("matmul", "distance"):
        st["pairs"].launch([d["a"], d["b"], d["p"]], rows=case["m"], cols=case["n"], dim=case["k"])
        return [t["p"]]
    if kind == "matmul_train":
        p, m, k, n = st["pairs"], case["m"], case["k"], case["n"]
        p.launch([d["a"], d["b"], d["p"]], rows=m, cols=n, dim=k)
        p.launch([d["g"], d["b"], d["ga"]], rows=m, cols=k, dim=n, flags=S.SHAPE_TRANS_RIGHT)
        p.launch([d["a"], d["g"], d["gb"]], rows=k, cols=n, dim=m, flags=S.SHAPE_TRANS_LEFT)
        return [t["p"], t["ga"], t["gb"]]
    n, plan = st["n"], st["plan"]
    st["map"].launch([d["x"], d["m"]], n=n)
    st["scan"].launch([d["m"], d["s"]], n=n, flags=S.SHAPE_INCLUSIVE, segments=plan)
    st["sum"].launch([d["s"], d["r"]], n=n, segments=plan)
    S.check(S.lib().scl_adjoint_broadcast_segments(d["g"].ptr, d["gs"].ptr, d["off"].ptr, case["vectors"], n,
                                                   S.DTYPE_F32, 0))
    st["scan"].launch([d["gs"], d["gm"]], n=n, flags=S.SHAPE_INCLUSIVE | S.SHAPE_REVERSE, segments=plan)
    st["madj"].launch([d["x"], d["gm"], d["gx"]], n=n)
    return [t["s"], t["r"], t["gx"]]


def work(case):
    kind = case["kind"]
    size = {"float": 4, "double": 8, "int": 4}.get(case.get("dtype"), 4)
    if kind == "dot":  # x, y read, the product and the sum written
        return {"bytes": 3 * size * case["n"] + size, "flops": 2 * case["n"]}
    if kind == "scan_mod":  # x read, the sums and their remainders written
        return {"bytes": 12 * case["n"], "flops": 2 * case["n"]}
    if kind == "scan_train":
        return {"bytes": 4 * size * case["n"], "flops": 2 * case["n"]}
    if kind == "map_train":  # x, g read, the values and the gradient written
        return {"bytes": 4 * size * case["n"], "flops": 4 * case["n"]}
    if kind == "blur_train":
        px, taps = case["rows"] * case["cols"], (2 * case["r"] + 1) ** 2
        return {"bytes": 16 * px, "flops": 4 * taps * px}
    if kind == "sobel":
        px = case["rows"] * case["cols"]
        return {"bytes": 2 * px, "flops": 13 * px}
    if kind == "segments_train":
        if case["law"] == "log":
            mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        else:
            mean = (case["lo"] + case["hi"] - 1) / 2
        n = int(mean * case["vectors"])
        # x and each vector's gradient and offset read; the prefix sums, the
        # vectors' sums and the gradient written
        return {"bytes": 12 * n + 16 * case["vectors"], "flops": 7 * n}
    m, k, n = case["m"], case["k"], case["n"]
    if kind == "distance":
        return {"bytes": 4 * (m * k + k * n + m * n), "flops": 3 * m * k * n}
    if kind == "matmul":
        return {"bytes": 4 * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    return {"bytes": 8 * (m * k + k * n + m * n), "flops": 6 * m * k * n}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("scan_mod", "sobel") or case.get("dtype") == "int":
        return None  # whole numbers
    i = _inputs(case, seed)
    if kind == "dot":
        z = i["x"].double() * i["y"].double()
        # the Reduce is given the products as they were stored
        return [z, (i["x"] * i["y"]).double().sum().reshape(1)]
    if kind == "scan_train":
        s, gx = i["x"].double().cumsum(0), i["g"].double().flip(0).cumsum(0).flip(0)
        if not case["inclusive"]:
            s, gx = s - i["x"].double(), gx - i["g"].double()
        return [s, gx]
    if kind == "map_train":
        x = i["x"].double()
        return [x * x + 1, 2 * x * i["g"].double()]
    if kind == "blur_train":
        h, w, r = case["rows"], case["cols"], case["r"]
        x, g = i["x"].double().reshape(h, w), i["g"].double().reshape(h, w)
        mode = "replicate" if case["nearest"] else "constant"
        xp = torch.nn.functional.pad(x[None, None], (r, r, r, r), mode=mode)[0, 0]
        out, gp = torch.zeros_like(x), torch.zeros_like(xp)
        for dy in range(2 * r + 1):
            for dx in range(2 * r + 1):
                c = float(i["w"][dy, dx])
                out += c * xp[dy:dy + h, dx:dx + w]
                gp[dy:dy + h, dx:dx + w] += c * g
        if case["nearest"]:  # what the clamped border was read for
            gp[r] += gp[:r].sum(0)
            gp[r + h - 1] += gp[r + h:].sum(0)
            gp[:, r] += gp[:, :r].sum(1)
            gp[:, r + w - 1] += gp[:, r + w:].sum(1)
        return [out.reshape(-1), gp[r:r + h, r:r + w].reshape(-1)]
    if kind in ("matmul", "matmul_train"):
        a, b = i["a"].double(), i["b"].double()
        if kind == "matmul":
            return [a @ b]
        g = i["g"].double()
        return [a @ b, g @ b.T, a.T @ g]
    if kind == "distance":
        a, bt = i["a"].double(), i["b"].double().T.contiguous()
        return [torch.cat([(a[r:r + 16, None, :] - bt[None]).abs().sum(2) for r in range(0, a.shape[0], 16)])]
    # segments: sums within each vector from one running sum
    x, off, n = i["x"].double(), i["off"], i["n"]
    lens = off[1:] - off[:-1]
    run_sum = torch.zeros(n + 1, device="cuda", dtype=torch.float64)
    torch.cumsum((x * x + 1), 0, out=run_sum[1:])
    s = run_sum[1:] - torch.repeat_interleave(run_sum[off[:-1]], lens)
    del run_sum
    run_sum = torch.zeros(n + 1, device="cuda", dtype=torch.float64)
    torch.cumsum(s, 0, out=run_sum[1:])
    # (long vectors' sums of prefix sums are large: their difference loses
    # nothing that matters next to single precision)
    r = run_sum[off[1:]] - run_sum[off[:-1]]
    del run_sum
    left = torch.repeat_interleave(off[1:], lens) - torch.arange(n, device="cuda")
    gx = 2 * x * torch.repeat_interleave(i["g"].double(), lens) * left
    return [s, r, gx]
