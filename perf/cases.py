"""The work that programs have this library do, as cases that can be timed.

Every case names a kind of call (`op`) and its sizes:

  call    one picture in device memory, the whole chain from its CU lists
          (a decoder that hands over each picture as it is reconstructed)
  plans   many device pictures whose side information is resident, in one
          batched execution (an encoder's repeated trials, re-filtering)
  fresh   the same batch with the deblocking side information derived from
          the CU lists and the motion on every execution (a decoder of many
          streams that keeps its lists on the device)
  host    pictures in pinned host memory: uploads, chain and downloads of the
          whole call (a decoder that reconstructs on the host)
  serve   requests of several picture sizes submitted to the server at once
          and waited for (a service with many concurrent streams)
  alf     an encoder's ALF decisions of one picture: luma, then Cb and Cr,
          then the cross-component filters
  sao     an encoder's SAO decision of one picture and its chroma merge
  recon   the steps either side of the chain for one picture: forward luma
          map, chroma residual scales, chroma residual add, output dump

Device pictures are filtered in place, so a pass first puts the unfiltered
samples back, as the reconstruction of the next picture would write them;
pictures in host memory and the server's pictures are filtered again as they
are, since their time lies in the link and the launches.  The outputs are
whole numbers: samples, decisions and byte dumps, equal on every machine.
"""
import importlib.util
import os
import pathlib
import sys

import numpy as np
import torch

ROOT = pathlib.Path(os.getcwd())


def _package():
    if "oxideav_h266_b200" not in sys.modules:
        pkg = ROOT / "oxideav-h266_b200"
        spec = importlib.util.spec_from_file_location("oxideav_h266_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["oxideav_h266_b200"] = mod
        spec.loader.exec_module(mod)
    from oxideav_h266_b200 import abi, native, workloads

    return abi, native, workloads


abi, native, W = _package()

_SHARED = {}


def _context():
    """One context on one stream for the whole program, as a decoder keeps."""
    if "ctx" not in _SHARED:
        torch.cuda.set_device(0)
        stream = torch.cuda.Stream()
        torch.cuda.set_stream(stream)
        ctx = native.Context(0)
        ctx.set_stream(stream.cuda_stream)
        _SHARED["stream"], _SHARED["ctx"] = stream, ctx
    return _SHARED["ctx"]


def _server():
    if "server" not in _SHARED:
        _SHARED["server"] = native.Server(0, max_batch=64, memory_budget=40 << 30)
    return _SHARED["server"]


def _case(name, op, w, h, n=1, bd=10, ctb=7, cfi=1, part="quad", inter=0.5, aps=4, lmcs=True, cc=True, tiles=False):
    return {"name": name, "op": op, "w": w, "h": h, "n": n, "bd": bd, "ctb": ctb, "cfi": cfi, "part": part,
            "inter": inter, "aps": aps, "lmcs": lmcs, "cc": cc, "tiles": tiles}


def listed():
    return [
        # the smallest picture a decoder hands over: all intra, one APS, no LMCS or CC-ALF (launches and latency)
        _case("call_416x240_8b", "call", 416, 240, bd=8, inter=0.0, aps=1, lmcs=False, cc=False),
        # one full-HD picture at a time from the decoder, every tool on
        _case("call_1080p10", "call", 1920, 1080),
        # the throughput of resident full-HD pictures (the benchmark's picture)
        _case("plans_1080p10_x16", "plans", 1920, 1080, n=16),
        # the same pictures, their edges derived from the CU lists on every execution
        _case("fresh_1080p10_x16", "fresh", 1920, 1080, n=16),
        # multi-type-tree partitions down to 4 samples with transform splits and sub-block motion
        _case("fresh_mtt_1080p10_x8", "fresh", 1920, 1080, n=8, part="mtt", aps=2),
        # 2160p intra pictures, 4x2 tiles that are not filtered across: the largest call
        _case("plans_2160p10_tiles_x8", "plans", 3840, 2160, n=8, inter=0.0, aps=1, lmcs=False, cc=False, tiles=True),
        # 4:4:4 screen and studio content
        _case("plans_444_1080p10_x4", "plans", 1920, 1080, n=4, cfi=3, aps=2),
        # reconstruction on the host: the link in both directions and the preparation of the lists
        _case("host_1080p10_x16", "host", 1920, 1080, n=16),
        # 12 requests of three picture sizes at once
        _case("serve_mix_x12", "serve", 1920, 1080, n=12, inter=0.0, aps=1, lmcs=False, cc=False),
        # an encoder's loop-filter decisions for one full-HD picture
        _case("alf_1080p10", "alf", 1920, 1080, aps=1),
        _case("sao_1080p10", "sao", 1920, 1080, aps=1),
        # the steps around the chain for one full-HD picture
        _case("recon_1080p10", "recon", 1920, 1080, aps=1),
    ]


# most luma samples of one pass, by kind: none costs more than the largest listed case
_MOST = {"call": 9e6, "plans": 5e7, "fresh": 3.3e7, "host": 1.6e7, "serve": 2.5e7, "alf": 4.2e6, "sao": 9e6,
         "recon": 9e6}


def draw(rng):
    op = rng.choice(sorted(_MOST))
    single = op in ("call", "alf", "sao", "recon")
    enc = op in ("alf", "sao", "recon")
    cfi = 1 if enc or op in ("host", "serve") else rng.choice((1, 1, 1, 2, 3))
    part = "quad" if enc or op in ("host", "serve") else rng.choice(("quad", "quad", "mtt"))
    most = _MOST[op] / (4 if cfi != 1 or part == "mtt" else 1)
    if rng.random() < 0.35:  # the sizes that are broadcast and streamed
        w, h = rng.choice(((416, 240), (832, 480), (1280, 720), (1920, 1080), (2560, 1440), (3840, 2160)))
    else:
        step = rng.choice((2, 8, 8, 16))
        w = int(128 * 2 ** rng.uniform(0, 4.9)) // step * step
        h = max(96, int(w * rng.uniform(0.4, 0.8))) // step * step
    if part == "mtt":
        w, h = w // 8 * 8, h // 8 * 8
    while w * h > most:
        w, h = max(128, w // 16 * 8), max(96, h // 16 * 8)
    n = 1 if single else max(1, min(64, int(most / (w * h) * 2 ** -rng.uniform(0, 3))))
    c = _case("", op, w, h, n=n, bd=rng.choice((8, 10, 10, 12)), ctb=rng.choice((5, 6, 7, 7)), cfi=cfi, part=part,
              inter=rng.choice((0.0, 0.3, 0.5, 0.8)), aps=rng.choice((1, 2, 4)), lmcs=enc or rng.random() < 0.6,
              cc=enc or rng.random() < 0.6, tiles=not enc and part == "quad" and rng.random() < 0.25)
    del c["name"]
    return c


def _tiles(case, w, h):
    """4 x 2 uniform tiles, in CTBs, where the picture has as many."""
    ctb = 1 << case["ctb"]
    wc, hc = -(-w // ctb), -(-h // ctb)
    if not case["tiles"] or wc < 4 or hc < 2:
        return None
    q, r = -(-wc // 4), -(-hc // 2)
    return [q, q, q, wc - 3 * q] if wc > 3 * q else [1, 1, 1, wc - 3], [r, hc - r]


def _picture(case, seed, w, h):
    if case["part"] == "mtt":
        pic, fa = W.stress_workload(seed, w, h, case["bd"], case["ctb"])
    else:
        pic, fa = W.make_workload(seed, w, h, case["bd"], case["ctb"], inter_frac=case["inter"],
                                  n_luma_aps=case["aps"], n_chroma_alt=4 if case["op"] == "alf" else 2,
                                  ccalf=case["cc"], lmcs=case["lmcs"], tiles=_tiles(case, w, h))
    return W.with_chroma_format(pic, fa, case["cfi"], seed) if case["cfi"] != 1 else (pic, fa)


def _sizes(case):
    """(w, h) of each picture of the pass."""
    w, h = case["w"], case["h"]
    if case["op"] != "serve":
        return [(w, h)] * case["n"]
    mix = ((w, h), (max(128, w // 16 * 8), max(96, h // 16 * 8)), (w, h), (max(128, w // 32 * 16), max(96, h // 32 * 16)))
    return [mix[i % 4] for i in range(case["n"])]


def _items(case, seed):
    """Pictures and arguments of the pass: up to four different ones of a size, repeated over the batch."""
    most = 2 if case["part"] == "mtt" or case["w"] * case["h"] > 4e6 else 4
    made, items, seen = {}, [], {}
    for i, size in enumerate(_sizes(case)):
        k = seen.get(size, 0)
        seen[size] = k + 1
        key = (size, k % most)
        if key not in made:
            made[key] = _picture(case, seed * 64 + len(made), *size)
        items.append(made[key])
    return items


def _flat(pics, device):
    """All planes of `pics` in one int16 tensor, each at a 256-byte boundary, and their places."""
    at, end = [], 0
    for p in pics:
        planes = []
        for a in p.planes():
            planes.append((end, a.shape))
            end += -(-a.size // 128) * 128
        at.append(planes)
    host = torch.zeros(max(end, 1), dtype=torch.int16, pin_memory=device is None)
    flat = host.numpy()
    for p, planes in zip(pics, at):
        for a, (o, _) in zip(p.planes(), planes):
            flat[o:o + a.size] = np.ascontiguousarray(a).view(np.int16).reshape(-1)
    return (host if device is None else host.to(device)), at


def _views(flat, at, bd):
    out = []
    for planes in at:
        v = [flat[o:o + s[0] * s[1]].view(s) for o, s in planes]
        if flat.is_cuda:
            out.append(native.DevicePicture(*v, bd))
        else:
            out.append(W.PictureData(*[t.numpy().view(np.uint16) for t in v], bd))
    return out


def _noisy(pic, seed):
    """The encoder's original: the picture plus noise in [-6, 6]."""
    rng = np.random.Generator(np.random.PCG64(seed + 17))
    mx = (1 << pic.bit_depth) - 1
    planes = [np.clip(p.astype(np.int64) + rng.integers(-6, 7, size=p.shape), 0, mx).astype(np.uint16)
              for p in pic.planes()]
    return W.PictureData(*planes, pic.bit_depth)


def prepare(case, seed):
    ctx = _context()
    op = case["op"]
    items = _items(case, seed)
    pics, fas = [p for p, _ in items], [f for _, f in items]
    st = {"op": op, "ctx": ctx, "fas": fas, "bd": case["bd"], "ctb": case["ctb"]}
    if op == "host":
        st["work"], at = _flat(pics, None)
        st["pics"] = _views(st["work"], at, case["bd"])
        st["call"] = ctx.batch_call(st["pics"], fas)
        return st
    st["source"], at = _flat(pics, "cuda")
    st["work"] = st["source"].clone()
    st["pics"] = _views(st["work"], at, case["bd"])
    if op in ("plans", "fresh", "serve"):
        st["plans"] = [ctx.plan(p, f, device_sideinfo=op == "fresh") for p, f in items]
    if op == "serve":
        st["server"] = _server()
    if op in ("alf", "sao"):
        src = _noisy(pics[0], seed)
        st["src_flat"], src_at = _flat([src], "cuda")
        st["src"] = _views(st["src_flat"], src_at, case["bd"])[0]
        st["grid"] = (-(-case["w"] // (1 << case["ctb"])), -(-case["h"] // (1 << case["ctb"])))
        st["pre_luma"] = _views(st["source"], at, case["bd"])[0].luma
    if op == "recon":
        cus = fas[0].cus
        rects = np.zeros(len(cus), dtype=abi.RECT)
        for f in ("x", "y", "w", "h"):
            rects[f] = cus[f]
        # one chroma scale per 64x64 luma region, the unit that shares it
        ys, xs = np.mgrid[0:case["h"]:64, 0:case["w"]:64]
        cvs = np.zeros(xs.size, dtype=abi.CVS_BLOCK)
        cvs["x_cu_cb"], cvs["y_cu_cb"] = xs.reshape(-1), ys.reshape(-1)
        cvs["avail_l"], cvs["avail_t"] = cvs["x_cu_cb"] > 0, cvs["y_cu_cb"] > 0
        rng = np.random.Generator(np.random.PCG64(seed + 1))
        blocks = np.zeros(2 * len(cus), dtype=abi.RES_BLOCK)
        for f in ("x", "y", "w", "h"):
            blocks[f] = np.repeat(cus[f] // 2, 2)
        blocks["w"] = np.minimum(blocks["w"], case["w"] // 2 - blocks["x"])
        blocks["h"] = np.minimum(blocks["h"], case["h"] // 2 - blocks["y"])
        blocks["plane"] = np.tile([1, 2], len(cus))
        blocks["var_scale"] = rng.integers(1024, 4096, len(blocks))
        area = blocks["w"].astype(np.uint64) * blocks["h"]
        blocks["res_offset"] = np.concatenate([[0], np.cumsum(area)[:-1]])
        st["rects"], st["cvs"], st["blocks"] = rects, cvs, blocks
        st["res"] = torch.tensor(rng.integers(-64, 65, int(area.sum()), dtype=np.int32), device="cuda")
        st["crop"] = (0, 0, case["w"], case["h"])
        samples = case["w"] * case["h"] + 2 * (case["w"] // 2) * (case["h"] // 2)
        st["dump"] = torch.zeros(samples * (1 if case["bd"] == 8 else 2), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return st


def run(st):
    op, ctx, pics = st["op"], st["ctx"], st["pics"]
    if op == "host":
        st["call"].run()
        return st["work"]
    if op == "serve":
        srv = st["server"]
        tickets = [srv.submit(plan, pic) for plan, pic in zip(st["plans"], pics)]
        for t in tickets:
            srv.wait(t)
        return st["work"]
    if op == "sao":  # the pre-SAO picture is only read
        out = native.sao_decide_picture(ctx, st["src"], pics[0], ctb_log2=st["ctb"], bit_depth=st["bd"])
        merged, where = native.sao_chroma_merge(ctx, st["src"], pics[0], out, *st["grid"], bit_depth=st["bd"],
                                                ctb_log2=st["ctb"])
        return {"decided": out.view(np.uint8), "merged": merged.view(np.uint8), "map": where}
    st["work"].copy_(st["source"])
    if op == "call":
        ctx.apply_in_loop_filters(pics[0], st["fas"][0])
        return st["work"]
    if op in ("plans", "fresh"):
        ctx.execute_plans(st["plans"], pics)
        return st["work"]
    if op == "alf":
        src, rec, fa = st["src"], pics[0], st["fas"][0]
        aps, how = fa.apses[0], dict(ctb_log2=st["ctb"], bit_depth=st["bd"])
        dec, _ = native.alf_decide_and_apply(ctx, src, rec, aps, **how)
        for component in (1, 2):
            native.chroma_alf_decide(ctx, src, rec, dec, aps, component=component, cc=False, **how)
        for component in (1, 2):
            native.chroma_alf_decide(ctx, src, rec, dec, aps, component=component, cc=True, pre_luma=st["pre_luma"],
                                     **how)
        return {"decided": dec.view(np.uint8), "rec": st["work"]}
    assert op == "recon"
    pic, fa = pics[0], st["fas"][0]
    native.lmcs_forward_map_luma_rects(ctx, pic, fa.lmcs, st["rects"])
    scales = native.lmcs_chroma_var_scale(ctx, pic, fa.lmcs, fa.lmcs_min_bin, fa.lmcs_max_bin, 1 << st["ctb"],
                                          st["cvs"])
    native.lmcs_add_chroma_residual(ctx, pic, st["bd"], st["res"], st["blocks"])
    native.output_convert(ctx, pic, st["crop"], 1, st["bd"], dst=st["dump"])
    return {"scales": scales.astype(np.int64), "picture": st["work"], "dump": st["dump"]}


def work(case):
    """Each 16-bit plane read once and written once; the CU lists and CTB parameters are about a tenth of that at most
    and are left out.  All arithmetic is on whole numbers."""
    luma = sum(w * h for w, h in _sizes(case))
    samples = luma * {1: 1.5, 2: 2.0, 3: 3.0}[case["cfi"]]
    if case["op"] == "sao":
        b = 2 * 2 * samples  # original and reconstruction read
    elif case["op"] == "alf":
        b = 3 * 2 * samples + 2 * luma  # original and reconstruction read, reconstruction written, pre-ALF luma read
    elif case["op"] == "recon":
        b = 4 * luma + 0.5 * luma * (4 + 4) + (2 + (1 if case["bd"] == 8 else 2)) * samples
    else:
        b = 2 * 2 * samples
    return {"bytes": float(b), "flops": 0.0}
