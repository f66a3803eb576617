"""The work that is timed: linears of one decoder layer through the operators and the GPU binding, and the trellis converter.

A case is one of
  linear   one linear of the format's operator (`formats.*.linear`), which routes itself by row count: the decode kernels,
           the tensor-core routes for more rows
  layer    the linears of one decoder layer. Up to 8 rows on q3 and nvfp4: q+k+v as a group, o, gate+up as a group, down.
           More rows, and trellis: the fused objects of an artifact (query_key_value, o, gate_up, down); gate_up runs as the
           paired SwiGLU region where the format's prefill has one
  region   the paired gate/up SwiGLU region of a prefill alone
  convert  a dense weight to a trellis object (`TrellisConverter.quantize`)
Layers are `hidden` wide with `inter` gate and up rows, as many query rows as `hidden` and `kv` key and value rows. Everything
of a pass is queued on one stream with programmatic dependent launch, as a decode step or a prompt chunk is.
"""

import math

import torch

from euhedral_b200 import layouts, synthetic
from euhedral_b200.formats import GroupedLinearFormat, LinearLaunch, Nvfp4Format, TensorHandle, TrellisFormat, TrellisSettings
from euhedral_b200.gpu import CudaGpuMemory
from euhedral_b200.trellis_convert import TrellisConverter, words_per_tile

SIGMA = 0.02          # standard deviation of the weights
DECODE_ROWS = 8       # most rows of one decode launch
MOST_FLOPS = 2.0 * 32768 * 34816 * 5120


def listed():
    return [
        # the smallest linear of a layer at one token: launch latency and host work
        {"name": "nvfp4 k, 1 row", "op": "linear", "format": "nvfp4", "rows": 1, "n": 1024, "k": 5120, "exact": False},
        # decode of one token, three formats and row counts: a plain step, a step that verifies drafted tokens
        {"name": "q3 layer, 1 row", "op": "layer", "format": "q3", "rows": 1, "hidden": 5120, "kv": 1024, "inter": 17408, "exact": False},
        {"name": "nvfp4 layer, 5 rows", "op": "layer", "format": "nvfp4", "rows": 5, "hidden": 5120, "kv": 1024, "inter": 17408, "exact": False},
        {"name": "trellis layer, 1 row", "op": "layer", "format": "trellis", "words": 48, "rows": 1, "hidden": 5120, "kv": 1024, "inter": 17408, "exact": False},
        # sizes that no tile divides, table-indexed scales
        {"name": "sd4 ragged, 3 rows", "op": "linear", "format": "sd4", "rows": 3, "n": 11024, "k": 4224, "exact": False},
        # a few sequences at once, every row with the bits of its own one-row call
        {"name": "q3 gate_up, 24 rows exact", "op": "linear", "format": "q3", "rows": 24, "n": 34816, "k": 5120, "exact": True},
        {"name": "trellis ragged, 17 rows", "op": "linear", "format": "trellis", "words": 56, "rows": 17, "n": 8320, "k": 4224, "exact": True},
        # a batch of short prompts or many sequences: too few rows to fill the chip with output tiles
        {"name": "nvfp4 layer, 40 rows", "op": "layer", "format": "nvfp4", "rows": 40, "hidden": 5120, "kv": 1024, "inter": 17408, "exact": False},
        # prompt chunks
        {"name": "q3 layer, 600 rows", "op": "layer", "format": "q3", "rows": 600, "hidden": 4096, "kv": 1024, "inter": 14336, "exact": False},
        {"name": "trellis layer, 2048 rows", "op": "layer", "format": "trellis", "words": 64, "rows": 2048, "hidden": 5120, "kv": 1024, "inter": 17408, "exact": False},
        # the largest: a long prompt through the widest region of a layer
        {"name": "nvfp4 region, 32768 rows", "op": "region", "format": "nvfp4", "rows": 32768, "n": 34816, "k": 5120, "exact": False},
        # what the converter does with every weight matrix
        {"name": "convert 1024x1024, 3 bits", "op": "convert", "bits": 3.0, "n": 1024, "k": 1024},
    ]


def _size(rng, low, high, unit):
    """A multiple of `unit` between low and high, even over the logarithm."""
    return max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))) / unit) * unit)


def draw(rng):
    while True:
        op = rng.choice(["linear"] * 4 + ["layer"] * 4 + ["region", "convert"])
        if op == "convert":
            case = {"op": op, "bits": rng.choice([2.0, 2.5, 3.0, 3.5, 4.0]), "n": _size(rng, 256, 2048, 128), "k": _size(rng, 256, 2048, 128)}
            if case["n"] * case["k"] > 1.5e6:
                continue
            return case
        case = {"op": op, "format": rng.choice(["q3", "nvfp4", "nvfp4", "sd4", "trellis"])}
        rows = _size(rng, 1, 8, 1) if rng.random() < 0.4 else _size(rng, 1, 16384, 1)
        if op == "region":
            case["format"] = rng.choice(["q3", "nvfp4"])
            rows = _size(rng, 64, 32768, 1)
        if case["format"] == "trellis":
            case["words"] = rng.choice([32, 40, 48, 56, 64])
            rows = min(rows, 16384)
        case["rows"] = rows
        if op == "layer":
            case["hidden"] = _size(rng, 1024, 8192, 256)
            case["kv"] = 128 * rng.choice([4, 8, 16])
            case["inter"] = _size(rng, 2 * case["hidden"], 4 * case["hidden"], 256)
        else:
            # decode takes any multiple of 16 columns and of 128 values; the routes for more rows want whole tiles
            decode = rows <= DECODE_ROWS and case["format"] != "trellis"
            case["n"] = _size(rng, 512, 32768, 256 if op == "region" else 16 if decode else 128)
            case["k"] = _size(rng, 1024, 16384, 128 if decode or case["format"] in ("q3", "trellis") else 256)
        case["exact"] = 8 < rows <= 32 and rng.random() < 0.5
        if work(case)["flops"] <= MOST_FLOPS and work(case)["bytes"] <= 2e9:
            return case


def _objects(case):
    """(name, rows of the weight, K, paired) of every linear of a pass."""
    if case["op"] != "layer":
        return [("linear", case["n"], case["k"], case["op"] == "region")]
    h, kv, i = case["hidden"], case["kv"], case["inter"]
    if case["rows"] <= DECODE_ROWS and case["format"] != "trellis":
        return [("q", h, h, False), ("k", kv, h, False), ("v", kv, h, False), ("o", h, h, False), ("gate", i, h, False), ("up", i, h, False),
                ("down", h, i, False)]
    # a region needs the prefill route: q3 takes it from 33 rows, nvfp4 from 9; row-exact calls are plain linears
    paired = case["format"] != "trellis" and case["rows"] > (32 if case["format"] == "q3" else 8) and not case["exact"]
    return [("query_key_value", h + 2 * kv, h, False), ("o", h, h, False), ("gate_up", 2 * i, h, paired), ("down", h, i, False)]


def _segments(case, name):
    if name == "query_key_value":
        return [case["hidden"], case["hidden"] + case["kv"], case["hidden"] + 2 * case["kv"]]
    if name == "gate_up":
        return [case["inter"], 2 * case["inter"]]
    return None


def _weight_bytes(case, name, n, k):
    if case["format"] == "q3":
        return layouts.q3_algorithmic_bytes(n, k)
    if case["format"] == "nvfp4":
        return layouts.nvfp4_algorithmic_bytes(n, k)
    if case["format"] == "sd4":
        return layouts.nvfp4_algorithmic_bytes(n, k) - n * k // 32 + 16
    return layouts.trellis_algorithmic_bytes(n, k, case["words"], len(_segments(case, name) or [n]))


def work(case):
    if case["op"] == "convert":
        tiles = case["n"] * case["k"] // 256
        # per tile two passes of 256 positions over 65,536 states: a difference, its square added to a cost, a comparison
        return {"bytes": case["n"] * case["k"] * 4 + tiles * words_per_tile(case["bits"]) * 2 + 2 * (case["n"] + case["k"]),
                "flops": tiles * 2.0 * 256 * 65536 * 4}
    total, flops = 0, 0.0
    for name, n, k, paired in _objects(case):
        shared = name in ("k", "v", "up")   # the input is read with the first tensor of the group
        total += _weight_bytes(case, name, n, k) + (0 if shared else 2 * case["rows"] * k) + 2 * case["rows"] * (n // 2 if paired else n)
        flops += 2.0 * case["rows"] * n * k
    return {"bytes": total, "flops": flops}


def tolerance(case):
    if case["op"] == "convert":
        return "exact"   # the search is defined to the bit
    # BF16 outputs of FP32 sums: most equal, the rest one BF16 step (2^-8 of the value) away; the prefill of trellis rounds its
    # operands and products to BF16 on the way
    return {"rel": 4e-3, "max": 2e-2}


_session = {}


def _gpu():
    if not _session:
        _session["gpu"] = CudaGpuMemory()
        _session["stream"] = torch.cuda.Stream()
        _session["converter"] = TrellisConverter()
        _session["trellis"] = TrellisFormat(TrellisSettings.for_device(_session["gpu"].multiprocessor_count()))
        _session["nvfp4"], _session["sd4"], _session["q3"] = Nvfp4Format(), Nvfp4Format(sd4=True), GroupedLinearFormat()
    return _session


def _sd4(plain, n, k):
    """The tensor with its block scales drawn from a table of 16 of its own codes."""
    at, blocks = layouts.nvfp4_scale_offset(n, k), n * k // 16
    codes = plain[at:at + blocks].int()
    table = torch.quantile(codes[:1 << 20].float(), torch.linspace(0.0, 1.0, 16, device=codes.device)).round().int()
    index = torch.searchsorted((table[1:] + table[:-1]).float() / 2, codes.float())
    out = torch.zeros(layouts.nvfp4_sd4_byte_size(n, k), dtype=torch.uint8, device=plain.device)
    out[:n * k // 2] = plain[:n * k // 2]
    out[at:at + blocks // 2] = (index[0::2] | index[1::2] << 4).to(torch.uint8)
    end = layouts.nvfp4_sd4_table_offset(n, k)
    out[end:end + 16] = table.to(torch.uint8)
    out[end + 16:end + 20] = plain[layouts.nvfp4_trailer_offset(n, k):][:4]
    return out


def _weights(case, name, n, k, seed):
    """(tensors to keep, TensorHandles) of one weight object."""
    if case["format"] == "trellis":
        ends = _segments(case, name) or [n]
        payload, suh, svh, _ = synthetic.trellis_object(n, k, case["words"], seed, segments=len(ends), device="cuda")
        keep = [payload, suh, svh, torch.tensor(ends, dtype=torch.int32, device="cuda")]
        return keep, [TensorHandle(name, tuple(t.shape), t.data_ptr(), t.numel() * t.element_size()) for t in keep]
    dense = synthetic.gaussian(n, k, seed, SIGMA, device="cuda")
    blob = synthetic.q3_tensor(dense) if case["format"] == "q3" else synthetic.nvfp4_tensor(dense)
    if case["format"] == "sd4":
        blob = _sd4(blob, n, k)
    return [blob], [TensorHandle(name, (n, k), blob.data_ptr(), blob.numel())]


def prepare(case, seed):
    s = _gpu()
    if case["op"] == "convert":
        return {"convert": (synthetic.gaussian(case["n"], case["k"], seed, SIGMA, device="cuda"), case["bits"], seed % 65536)}
    gpu, fmt, rows = s["gpu"], s[case["format"]], case["rows"]
    keep, calls, outputs, grouped = [], [], {}, {}
    for i, (name, n, k, paired) in enumerate(_objects(case)):
        tensors, handles = _weights(case, name, n, k, seed * 16 + i)
        x = keep[-1] if name in ("k", "v", "up") else synthetic.bf16_rows(rows, k, seed * 16 + i, device="cuda")
        y = torch.zeros((rows, n // 2 if paired else n), dtype=torch.bfloat16, device="cuda")
        outputs[name] = y
        keep += [*tensors, x]
        w = handles[0]
        if paired:
            region = gpu.q3_mx_gate_up_swiglu_bf16 if case["format"] == "q3" else gpu.nvfp4_native_gate_up_swiglu_bf16
            calls.append((region, (x.data_ptr(), w.device_address, y.data_ptr(), rows, k, n, w.byte_size)))
        elif name in ("q", "k", "v", "gate", "up"):
            group = grouped.setdefault(name in ("gate", "up"), ([], [], [], [], []))
            for values, value in zip(group, (x.data_ptr(), w.device_address, y.data_ptr(), n, w.byte_size)):
                values.append(value)
            if name in ("v", "up"):
                ins, weights, outs, widths, sizes = group
                calls.append((gpu.linear_group_bf16, ("q3" if case["format"] == "q3" else "nvfp4", ins, weights, outs, rows, k, widths, sizes)))
        else:
            launch = LinearLaunch(x.data_ptr(), y.data_ptr(), handles, rows, k, n, row_exact=case["exact"], segment_ends=_segments(case, name))
            if case["format"] == "trellis":
                need = fmt.scratch_bytes(gpu, rows, k, n, handles[1].shape[0], row_exact=case["exact"])
                keep.append(torch.empty(max(need, 256), dtype=torch.uint8, device="cuda"))
                launch.scratch, launch.scratch_bytes = keep[-1].data_ptr(), keep[-1].numel()
            calls.append((fmt.linear, (gpu, launch)))
    return {"gpu": gpu, "stream": s["stream"].cuda_stream, "exact": case["exact"], "calls": calls, "outputs": outputs, "keep": keep}


def run(state):
    if "convert" in state:
        made = _session["converter"].quantize(*state["convert"])
        return {"payload": made.payload, "suh": made.suh, "svh": made.svh, "scale": made.scale}
    with state["gpu"].submit(state["stream"], pdl=True, row_exact=state["exact"]):
        for call, arguments in state["calls"]:
            if call(*arguments) is False:
                raise RuntimeError("a route declined a linear of the case")
    return state["outputs"]
