"""What the performance of this framework is measured on: the calls that its users make, over the sizes they make
them with.

A serving process decodes weights on every forward: one call per weight through ``MPServe_cuda`` (the drop-in under
the vLLM plugin), a decoder layer at once through ``FusedDecoder``, or a rank's whole model through
``BucketDecodePlan``.  A compressor builds sidecars, one call per weight, with the weight on the GPU or, as the
reference's script has it, in host memory.  Weights are FP8-E4M3 with a scale per tensor, per channel or per
128 x 128 block, or AWQ INT4 with groups of 128 in one of three sidecar layouts.

Every result is a bit pattern that the format fixes, so every comparison is exact.  Weights are random-init
(N(0, 0.02), or Student-t(4) x 0.02 for the heavy tails that trained weights have), quantised as
``mpserve_b200.workloads`` does.
"""
import math

import torch

import MPServe_cuda
from mpserve_b200 import sidecar
from mpserve_b200 import workloads as wl
from mpserve_b200.api import BucketDecodePlan

RECT_KEYS = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_col_start_i32",
             "bucket_col_len_i32", "bucket_row_offsets_i32", "row_indices_i32", "bucket_thread_startbit_u32",
             "bucket_bit_base_i64")
BY_SCALE_KEYS = ("bitstream_u64", "decode_syms_u16", "decode_lens_u8", "bucket_table_i32", "bucket_group_offsets_i32",
                 "group_rows_i32", "group_col_start_i32", "bucket_thread_startbit_u32", "bucket_bit_base_i64")
SHARED_KEYS = ("bitstream_u64", "decode_syms_i16", "decode_nbits_u8", "scale_bit_base_i64", "chunk_startbit_rel_u32",
               "chunk_out_base_u32", "chunk_meta_u32", "chunk_scale_id_i32", "out_idx_i32", "stream_chunk_ofs_i64",
               "stream_chunk_ids_i32")
MODELS = {"llama3_8b": wl.LLAMA3_8B, "llama3_70b": wl.LLAMA3_70B}
GROUP = 128          # AWQ group size, and the side of an FP8 scale block


def fp8(name, n, m, scale, k, dist="normal"):
    return dict(name=name, kind="fp8", n=n, m=m, scale=scale, k=k, dist=dist)


def awq(name, layout, n, m, k=256):
    return dict(name=name, kind="awq", layout=layout, n=n, m=m, k=k)


def plan(name, model, tp, layers, fused=False):
    return dict(name=name, kind="plan", model=model, tp=tp, layers=layers, fused=fused, k=1024)


def build(name, fmt, n, m, scale="channel", k=1024, host=False, dist="normal"):
    return dict(name=name, kind="build", format=fmt, n=n, m=m, scale=scale, k=k, host=host, dist=dist)


def listed():
    return [
        # one weight per call, as the plugin decodes: the smallest weight of the size sweep (a launch and its host side) ...
        fp8("fp8_smallest_128x256", 128, 256, "channel", 1024),
        # ... a lone square projection with one scale: few buckets, latency of a sub-stream counts ...
        fp8("fp8_tensor_scale_4096x4096", 4096, 4096, "tensor", 1024),
        # ... rows of no convenient length, heavy tails, the reference builder's default of 256 sub-streams ...
        fp8("fp8_ragged_2047x3000", 2047, 3000, "channel", 256, "student_t"),
        # ... and an MLP weight with per-channel scales, the ordinary large call of an 8B model
        fp8("fp8_channel_14336x4096", 14336, 4096, "channel", 1024),
        # one decoder layer into its fused qkv / gate_up weights, one launch
        plan("layer_8b_fused", "llama3_8b", 1, 1, fused=True),
        # a tensor-parallel rank's share of nine layers of the 70B model in one launch: the largest
        plan("shards_70b_tp8_9_layers", "llama3_70b", 8, 9),
        # INT4 weights in the three layouts
        awq("awq_by_scale_14336x4096", "by_scale", 14336, 4096),
        awq("awq_bucket_4096x4096", "bucket", 4096, 4096),
        awq("awq_shared_4096x4096", "shared", 4096, 4096),
        # the compressor: an MLP weight already on the GPU, a key/value projection handed over in host memory as the
        # reference's script does, and an INT4 weight
        build("build_fp8_14336x4096", "fp8", 14336, 4096),
        build("build_fp8_host_1024x4096", "fp8", 1024, 4096, host=True),
        build("build_awq_by_scale_4096x4096", "by_scale", 4096, 4096, k=256),
    ]


def _between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _width(rng, low, high):
    """Columns: mostly a multiple of 128 as hidden sizes are, or of 16, sometimes any number."""
    step = rng.choice((128, 128, 128, 16, 16, 1))
    return max(step, _between(rng, low, high) // step * step)


def draw(rng):
    kind = rng.choice(("fp8", "fp8", "fp8", "plan", "awq", "awq", "build", "build"))
    if kind == "fp8":
        n, m = _between(rng, 64, 16384), _width(rng, 256, 14336)
        scale = rng.choice(("channel", "channel", "tensor", "block"))
        if scale == "block":
            n, m = max(1, n // GROUP) * GROUP, max(1, m // GROUP) * GROUP
        return fp8(None, n, m, scale, rng.choice((256, 1024, 1024)), rng.choice(("normal", "normal", "student_t")))
    if kind == "plan":
        if rng.random() < 0.5:   # a layer has 0.22 G (8B) or 0.86 G (70B) elements; at most what the largest listed case has
            return plan(None, "llama3_8b", rng.choice((1, 2, 4)), rng.randint(1, 4), fused=rng.random() < 0.5)
        tp = rng.choice((2, 4, 8))
        return plan(None, "llama3_70b", tp, rng.randint(1, tp), fused=rng.random() < 0.5)
    if kind == "awq":
        layout = rng.choice(("by_scale", "bucket", "shared"))
        n, m = _between(rng, 64, 14336 if layout == "by_scale" else 4096), _between(rng, 256, 4096) // GROUP * GROUP
        return awq(None, layout, n, m, rng.choice((256, 256, 1024)))
    fmt = rng.choice(("fp8", "fp8", "by_scale"))
    host = rng.random() < 0.3
    n = _between(rng, 256, 4096 if host or fmt != "fp8" else 14336)
    m = _between(rng, 256, 4096) // GROUP * GROUP if fmt != "fp8" else _width(rng, 256, 4096)
    return build(None, fmt, n, m, rng.choice(("channel", "tensor")), rng.choice((256, 1024)), host, rng.choice(("normal", "student_t")))


# ---- inputs -----------------------------------------------------------------------------------------

def _fp8_weight(n, m, seed, scale, dist):
    return wl.quantize_fp8(wl.random_weight(n, m, seed, dist, device="cuda"), scale, (GROUP, GROUP))


def _awq_weight(n, m, seed):
    return wl.quantize_awq(wl.random_weight(n, m, seed, "normal", device="cuda"), GROUP)


def _shuffled(n, m, seed, dist, within):
    """A weight to compress.  How many tables and code bits a sidecar has depends on the weight, so the weights of two
    seeds are the same up to the order of the elements in every run of ``within`` columns: then the two sidecars
    differ in all that depends on an element's place and have the same shapes."""
    w = wl.random_weight(n, m, 7, dist, device="cuda").view(n, m // within, within)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    order = torch.rand(w.shape, generator=g, device="cuda").argsort(dim=2)
    return w.gather(2, order).view(n, m)


def _fp8_sidecar(c, k):
    return MPServe_cuda.huffman_build_fp8_decode_tables(c.bf16, c.fp8_u8, c.scales_u16, max_len=7, threads_per_block=k)


def _shards(case):
    """[layer][(name, n, m)] of what the plan decodes."""
    cfg = MODELS[case["model"]]
    one = [(name, *wl.tp_shard_shape(name, n, m, case["tp"])) for name, n, m in wl.layer_linears(cfg)]
    return [one] * case["layers"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fp8":
        n, m = case["n"], case["m"]
        c = _fp8_weight(n, m, seed, case["scale"], case["dist"])
        art = _fp8_sidecar(c, case["k"])
        args = (c.fp8_u8, *(art[key] for key in RECT_KEYS), n, m, 7)
        return lambda: MPServe_cuda.huffman_decode_fp8(*args)
    if kind == "plan":
        groups, entries = [], []
        for li, layer in enumerate(_shards(case)):
            weights = []
            for wi, (_, n, m) in enumerate(layer):
                c = _fp8_weight(n, m, seed * 1009 + li * 16 + wi, "channel", "normal")
                art = _fp8_sidecar(c, case["k"])
                weights.append((c.fp8_u8, {key: art[key] for key in RECT_KEYS}))
            q, k, v, o, gate, up, down = weights
            groups += [[q, k, v], [o], [gate, up], [down]]
            entries += [(ctx, art, None) for ctx, art in weights]
        return (sidecar.FusedDecoder(groups) if case["fused"] else BucketDecodePlan(entries)).decode
    if kind == "awq":
        n, m, k = case["n"], case["m"], case["k"]
        c = _awq_weight(n, m, seed)
        if case["layout"] == "shared":
            art = MPServe_cuda.huffman_build_awq_decode_tables(c.bf16, c.int4_u8, c.scales_u16, max_len=11)
            args = (*(art[key] for key in SHARED_KEYS), n * m, 11)
            return lambda: MPServe_cuda.huffman_decode_awq_shared_table(*args)
        if case["layout"] == "bucket":
            art = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables(c.bf16, c.int4_u8, c.scales_u16, max_len=11,
                                                                           threads_per_block=k)
            args = (c.int4_u8, *(art[key] for key in RECT_KEYS), n, m, 11)
            return lambda: MPServe_cuda.huffman_decode_awq_int4_bucket(*args)
        art = MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(c.bf16, c.int4_u8, c.scales_u16,
                                                                                max_len=11, threads=k, group_cap=1024)
        args = (c.int4_u8, *(art[key] for key in BY_SCALE_KEYS), n, m, 11, GROUP)
        return lambda: MPServe_cuda.huffman_decode_awq_int4_bucket_by_scale(*args)
    n, m, k, where = case["n"], case["m"], case["k"], "cpu" if case["host"] else "cuda"
    if case["format"] == "fp8":
        c = wl.quantize_fp8(_shuffled(n, m, seed, case["dist"], m), case["scale"])
        w = c.bf16.to(where), c.fp8_u8.to(where), c.scales_u16.to(where)
        return lambda: _stored(MPServe_cuda.huffman_build_fp8_decode_tables(*w, max_len=7, threads_per_block=k))
    c = wl.quantize_awq(_shuffled(n, m, seed, case["dist"], GROUP), GROUP)
    w = c.bf16.to(where), c.int4_u8.to(where), c.scales_u16.to(where)
    return lambda: _stored(MPServe_cuda.huffman_build_awq_int4_bucket_decode_tables_by_scale(*w, max_len=11, threads=k,
                                                                                             group_cap=1024))


SIGNED = {torch.uint16: torch.int16, torch.uint32: torch.int32, torch.uint64: torch.int64}


def _stored(art):
    """A sidecar in the types it is written to a file with, which has no wider unsigned ones."""
    return {key: t.view(SIGNED.get(t.dtype, t.dtype)) for key, t in art.items()}


def run(state):
    return state()


# ---- the work of a pass ------------------------------------------------------------------------------

def _fp8_bytes(n, m, scale, k, dist="normal"):
    """What the decode of an FP8 weight reads and writes: a byte in and two out per element, four bits of code, the
    start bits of every bucket, and a table of 320 bytes per context that a scale meets.  How many scales and contexts
    there are is an estimate from such weights: row maxima take some 95 different 16-bit values, 300 with heavy tails."""
    if scale == "tensor":
        tables, buckets, width = 1, -(-n // 128), m
    elif scale == "block":
        buckets, width = n * m // (GROUP * GROUP), GROUP
        tables = 75 * (1 - math.exp(-buckets / 75))
    else:
        most = 300 if dist == "student_t" else 95
        tables, width = most * (1 - math.exp(-n / most)), m
        buckets = tables + n // 256
    contexts = max(16.0, min(225.0, 25 * math.log2(2 + n * m / tables) - 125))
    return n * m * 3.5 + buckets * (min(k, 128 * width) + 260) * 4 + 4 * n + tables * contexts * 320


def work(case):
    kind, n, m = case["kind"], case.get("n"), case.get("m")
    if kind == "fp8":
        total = _fp8_bytes(n, m, case["scale"], case["k"], case["dist"])
    elif kind == "plan":
        total = sum(_fp8_bytes(a, b, "channel", case["k"]) for layer in _shards(case) for _, a, b in layer)
    else:
        layout = case["layout"] if kind == "awq" else case["format"]
        groups = n * m / GROUP
        scales = 450 * (1 - math.exp(-groups / 450))   # different scales among the groups of a Gaussian weight
        tables, codes = 16 * scales, n * m * 1.1       # of 2048 entries; some nine bits of code an element
        if layout == "shared":      # a chunk of 1.1 elements has 20 bytes of its own; an index of 4 bytes an element
            total = codes + n * m * (2 + 4 + 20 / 1.1) + tables * 2048 * 3
        elif layout == "bucket":    # a bucket per group: the start bits of its 128 sub-streams, 16 table numbers
            total = codes + n * m * 3 + groups * (129 * 4 + 64 + 24) + tables * 5120
        elif layout == "by_scale":
            total = codes + n * m * 3 + groups * 8 + (scales + groups / 1024) * (case["k"] + 20) * 4 + tables * 5120
        else:
            total = _fp8_bytes(n, m, case["scale"], case["k"], case["dist"])   # the same, read and written the other way round
    return {"bytes": int(total), "flops": 0}


def tolerance(case):
    return "exact"
