"""Performance cases of the match finders and the GPU entropy stage.

Each case is one call (or one chain of calls) that a program using this
library makes: through the `gcz` package on host buffers, or through its
device-pointer entry points on memory that torch owns.  `listed()` gives the
fixed cases, `draw(rng)` further ones of the same ranges, `prepare` what the
program holds before the call, `run` the call, `work` the bytes it cannot do
without.  All outputs are whole numbers or bytes.

Inputs come from the library's seeded generator (order-1 Markov text, copies
of earlier output, random bytes), in the benchmark's 40/40/20 mix or in a
text-like, a copy-heavy or a nearly incompressible one.
"""
import ctypes
import math
import os
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

PKG = os.path.join(os.getcwd(), "gpu-compressor_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import gcz  # noqa: E402

KIB, MIB, GIB = 1 << 10, 1 << 20, 1 << 30
SPAN = 8 * MIB  # generated at once by one thread; matches reach 64 KiB at most

# Markov / copy / random fractions.  "bench" is the benchmark's mix.
MIXES = {
    "bench": (0.4, 0.4, 0.2),
    "text": (0.8, 0.15, 0.05),
    "copies": (0.15, 0.8, 0.05),
    "dense": (0.1, 0.1, 0.8),
}


def listed():
    return [
        # The smallest request of the serving mix: 4 KiB of host bytes.
        {"name": "request_4k", "kind": "zstd_host", "bytes": 4 * KIB, "depth": 16, "mix": "bench"},
        # An ordinary small request: a few windows, the last one ragged.
        {"name": "request_200k", "kind": "zstd_host", "bytes": 200_003, "depth": 64, "mix": "bench"},
        # The Zstd L1 configuration: one 16 MiB buffer already on the device.
        {"name": "zstd_l1_16m", "kind": "zstd_device", "bytes": 16 * MIB, "depth": 16, "mix": "bench"},
        # The headline workload: Zstd L2 over 1 GiB on the device.
        {"name": "zstd_l2_1g", "kind": "zstd_device", "bytes": GIB, "depth": 64, "mix": "bench"},
        # The same from pinned host memory, copies included.
        {"name": "zstd_pinned_256m", "kind": "zstd_pinned", "bytes": 256 * MIB, "depth": 64, "mix": "bench"},
        # A batch of files of uneven sizes in one slab, window table on the device.
        {"name": "zstd_batch", "kind": "zstd_batch", "files": 96, "max_file": 16 * MIB, "sizes": 7, "depth": 16},
        # LZMA2 matches of a few ragged MiB on the device.
        {"name": "lzma2_3m", "kind": "lzma2_device", "bytes": 3 * MIB + 12_345, "mix": "text"},
        # The LZMA2 configuration: 1 GiB on the device, every position's match.
        {"name": "lzma2_1g", "kind": "lzma2_device", "bytes": GIB, "mix": "bench"},
        # One 128 MiB LZMA2 pipeline chunk from pinned memory, one bit per window back;
        # every other span is incompressible, which is what the bits sort out.
        {"name": "lzma2_triage_128m", "kind": "lzma2_triage", "bytes": 128 * MIB, "mix": "bench"},
        # A small buffer to finished Zstd frames, encoded on the GPU.
        {"name": "frames_1m", "kind": "frames_host", "bytes": MIB + 777, "level": 1, "mix": "text"},
        # Matches and frames of 256 MiB that is on the device and stays there.
        {"name": "frames_256m", "kind": "frames_device", "bytes": 256 * MIB, "depth": 64, "mix": "bench"},
        # The codec adapter on one 8 MiB pipeline chunk: libzstd codes the GPU's sequences on the host.
        {"name": "adapter_8m", "kind": "adapter", "bytes": 8 * MIB, "level": 1, "mix": "bench"},
    ]


def _size(rng, lo, hi):
    """Spread over the logarithm; most sizes are odd or ragged, some whole windows."""
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    if n >= 128 * KIB and rng.random() < 0.25:
        n = n // (64 * KIB) * (64 * KIB)
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["zstd_host", "zstd_device", "zstd_pinned", "zstd_batch", "lzma2_device", "lzma2_triage",
                       "frames_host", "frames_device", "adapter"])
    mix = rng.choice(sorted(MIXES))
    if kind == "zstd_batch":
        return {"kind": kind, "files": rng.randint(2, 96), "max_file": _size(rng, 64 * KIB, 16 * MIB),
                "sizes": rng.randint(0, 10**6), "depth": rng.choice([16, 64])}
    lo, hi = {"zstd_host": (KIB, 4 * MIB), "zstd_device": (64 * KIB, GIB), "zstd_pinned": (MIB, 256 * MIB),
              "lzma2_device": (64 * KIB, GIB), "lzma2_triage": (64 * KIB, 128 * MIB),
              "frames_host": (4 * KIB, 64 * MIB), "frames_device": (64 * KIB, 256 * MIB),
              "adapter": (64 * KIB, 8 * MIB)}[kind]
    case = {"kind": kind, "bytes": _size(rng, lo, hi), "mix": mix}
    if kind in ("zstd_host", "zstd_device", "zstd_pinned", "frames_device"):
        case["depth"] = rng.choice([16, 64])
    if kind in ("frames_host", "adapter"):
        case["level"] = rng.choice([1, 2])
    return case


def _fill(out, seed, mixes):
    """`out` filled span by span; span i has the mix mixes[i % len(mixes)]."""
    spans = range(0, out.size, SPAN)

    def one(i):
        o = spans[i]
        gcz.gen_synthetic(seed * 100_003 + i, min(SPAN, out.size - o), 8 * MIB, mixes[i % len(mixes)], out=out[o:o + SPAN])

    if len(spans) == 1:
        one(0)
    else:
        with ThreadPoolExecutor(os.cpu_count() or 4) as ex:
            list(ex.map(one, range(len(spans))))
    return out


def _file_sizes(case):
    sizes, _ = gcz.gen_file_sizes(case["sizes"], case["files"], 4 * KIB, case["max_file"])
    return [int(x) for x in sizes]


def _zeros(shape, dtype, pin=False):
    return torch.zeros(shape, dtype=dtype, pin_memory=True) if pin else torch.zeros(shape, dtype=dtype, device="cuda")


def _check(ctx, rc):
    if rc != 0:
        raise gcz.GczError(rc, gcz.L.gcz_last_error(ctx.handle).decode())


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "ctx": gcz.context(0), "case": case}
    if kind == "zstd_batch":
        sizes = _file_sizes(case)
        offsets, windows, slab_bytes = gcz.batch_layout(sizes)
        slab = np.zeros(slab_bytes, np.uint8)
        mixes = np.random.default_rng(seed).dirichlet([1, 1, 1], size=len(sizes))

        def one(i):
            o = int(offsets[i])
            gcz.gen_synthetic(seed * 100_003 + i, sizes[i], 8 * MIB, tuple(mixes[i]), out=slab[o:o + sizes[i]])

        with ThreadPoolExecutor(os.cpu_count() or 4) as ex:
            list(ex.map(one, range(len(sizes))))
        cap = sum(int(gcz.L.gcz_zstd_max_sequences(x)) for x in sizes)
        s.update(slab=torch.from_numpy(slab).cuda(), slab_bytes=slab_bytes, num_windows=len(windows), cap=cap,
                 windows=torch.from_numpy(windows.view(np.uint8).copy()).cuda(),
                 seqs=_zeros((cap, 4), torch.int32), offsets=_zeros(len(windows) + 1, torch.int64))
        return s
    n, mix = case["bytes"], MIXES[case["mix"]]
    nb = gcz.num_windows(n)
    s["n"] = n
    if kind in ("zstd_pinned", "lzma2_triage"):
        s["src"] = torch.empty(n, dtype=torch.uint8, pin_memory=True)
        _fill(s["src"].numpy(), seed, [mix] if kind == "zstd_pinned" else [(0.0, 0.0, 1.0), mix])
    else:
        s["src"] = torch.from_numpy(_fill(np.empty(n, np.uint8), seed, [mix]))
    if kind in ("frames_host", "adapter"):
        s["out_cap"] = int(gcz.L.gcz_zstd_frames_bound(n))
        s["out"] = np.zeros(s["out_cap"], np.uint8)
        s["sizes"] = np.zeros(nb, np.uint64)
        s["used"] = np.zeros(1, np.uint64)
        return s
    if kind == "lzma2_triage":
        s["has"] = np.zeros(nb, np.uint8)
        return s
    s["cap"] = int(gcz.L.gcz_zstd_max_sequences(n))
    if kind in ("zstd_host", "zstd_pinned"):
        s["seqs"] = _zeros((s["cap"], 4), torch.int32, pin=True)
        s["offsets"] = _zeros(nb + 1, torch.int64, pin=True)
        return s
    s["src"] = s["src"].cuda()
    if kind == "lzma2_device":
        s["packed"] = _zeros(n, torch.int32)
        s["has"] = _zeros(nb, torch.uint8)
        return s
    s["seqs"] = _zeros((max(s["cap"], 1), 4), torch.int32)
    s["offsets"] = _zeros(nb + 1, torch.int64)
    if kind == "frames_device":
        s["out_cap"] = int(gcz.L.gcz_zstd_frames_bound(n))
        s["out"] = _zeros(s["out_cap"], torch.uint8)
        s["frame_offsets"] = _zeros(nb + 1, torch.int64)
    return s


def run(s):
    kind, ctx, case = s["kind"], s["ctx"], s["case"]
    if kind in ("zstd_host", "zstd_pinned"):
        _check(ctx, gcz.L.gcz_zstd_match_find(ctx.handle, s["src"].data_ptr(), s["n"], case["depth"],
                                              s["seqs"].data_ptr(), s["cap"], s["offsets"].data_ptr()))
        return s["seqs"], s["offsets"]
    if kind == "lzma2_triage":
        _check(ctx, gcz.L.gcz_lzma2_match_find(ctx.handle, s["src"].data_ptr(), s["n"], gcz.LZMA2_SEARCH_DEPTH, None,
                                               s["has"].ctypes.data))
        return s["has"]
    if kind in ("frames_host", "adapter"):
        used = s["used"].ctypes.data_as(ctypes.POINTER(ctypes.c_size_t))
        if kind == "frames_host":
            rc = gcz.L.gcz_zstd_compress_frames_gpu(ctx.handle, s["src"].data_ptr(), s["n"], case["level"],
                                                    s["out"].ctypes.data, s["out_cap"], s["sizes"].ctypes.data, used)
        else:
            rc = gcz.L.gcz_zstd_compress_frames(ctx.handle, s["src"].data_ptr(), s["n"], case["level"], 0,
                                                s["out"].ctypes.data, s["out_cap"], s["sizes"].ctypes.data, used)
        _check(ctx, rc)
        return s["out"], s["sizes"], s["used"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "lzma2_device":
        ctx.lzma2_match_find_device(s["src"].data_ptr(), s["n"], gcz.LZMA2_SEARCH_DEPTH, s["packed"].data_ptr(),
                                    s["has"].data_ptr(), stream)
        return s["packed"], s["has"]
    if kind == "zstd_batch":
        ctx.zstd_match_find_batch_device(s["slab"].data_ptr(), s["slab_bytes"], s["windows"].data_ptr(),
                                         s["num_windows"], case["depth"], s["seqs"].data_ptr(), s["cap"],
                                         s["offsets"].data_ptr(), stream)
        return s["seqs"], s["offsets"]
    ctx.zstd_match_find_device(s["src"].data_ptr(), s["n"], case["depth"], s["seqs"].data_ptr(), s["cap"],
                               s["offsets"].data_ptr(), stream)
    if kind == "zstd_device":
        return s["seqs"], s["offsets"]
    ctx.zstd_encode_frames_device(s["src"].data_ptr(), s["n"], s["seqs"].data_ptr(), s["offsets"].data_ptr(),
                                  s["out"].data_ptr(), s["out_cap"], s["frame_offsets"].data_ptr(), stream)
    return s["seqs"], s["offsets"], s["out"], s["frame_offsets"]


# Output bytes per input byte, from the generator: ZSTD_Sequence records
# (16 bytes each) and finished frames.
RECORDS = {"bench": 0.32, "text": 0.51, "copies": 0.50, "dense": 0.045}
FRAMES = {"bench": 0.68, "text": 0.65, "copies": 0.40, "dense": 0.93}


def work(case):
    kind = case["kind"]
    if kind == "zstd_batch":
        n = sum(_file_sizes(case))
        return {"bytes": int(n * (1 + 0.30)), "flops": 0}
    n, mix, nb = case["bytes"], case["mix"], gcz.num_windows(case["bytes"])
    out = {"lzma2_device": 4 * n + nb, "lzma2_triage": nb, "frames_host": FRAMES[mix] * n + 8 * nb,
           "adapter": FRAMES[mix] * n + 8 * nb, "frames_device": (RECORDS[mix] + FRAMES[mix]) * n + 16 * nb}
    return {"bytes": int(n + out.get(kind, RECORDS[mix] * n + 8 * nb)), "flops": 0}
