"""Variant sweep and dispatch-table generator.

Counterpart of the reference's ``tools/grid_search.py`` (constraint pruning ``:89-116``, register / spill
parsing ``:124-151``, per-configuration timeout, CSV ``:170-251``) for the run-time variants of this library:
instead of recompiling one binary per macro combination it walks the compiled variant list
(``siglip_b200/csrc/sl8_variants.h``) through ``sl8_set_variant``, times every admissible variant on the
seeded synthetic operands of ``siglip_b200/synth.py`` over an M ladder (eight points per octave up to 16 images: a few
rows more can cost a whole round of tiles) from captured graphs (a Python loop takes longer than a small layer), writes one CSV row per
(layer, shape, variant) and turns the CSV into the table ``pick_variant`` (``sl8_api.cu``) consults:
``siglip_b200/csrc/sl8_dispatch_table.h``.

    python -m siglip_b200.sweep --shapes so400m,b16 --out siglip_b200/sweeps/b200.csv     # needs a B200
    python -m siglip_b200.sweep --emit-table siglip_b200/sweeps/b200.csv                   # CPU only

A variant that trips a bounded device wait is recorded as ``timeout`` (the kernel returns, the handle is
re-created) instead of hanging the sweep; that is this library's form of grid_search's per-run timeout.
"""
from __future__ import annotations

import argparse
import csv
import math
import random
import re
import statistics
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
TABLE_HEADER = PKG / "csrc" / "sl8_dispatch_table.h"
OPS = {"pe": 0, "fc1": 1, "fc2": 2}
OP_NAMES = {v: k for k, v in OPS.items()}
OP_ENUM = {0: "SL8_OP_PATCH_EMBED", 1: "SL8_OP_FC1_GELU", 2: "SL8_OP_FC2_RESIDUAL"}

# (layer, N, K, rows per image): the SigLIP-So400m/14 and SigLIP-B/16 layer shapes.
SHAPE_SETS = {
    "so400m": [("pe", 1152, 588, 729), ("fc1", 4304, 1152, 729), ("fc2", 1152, 4304, 729)],
    "b16": [("pe", 768, 768, 196), ("fc1", 3072, 768, 196), ("fc2", 768, 3072, 196)],
}
CSV_FIELDS = ["op", "M", "N", "K", "variant", "cta_group", "tile_n", "tile_k", "stages", "epi_warps", "staging_buffers",
              "regs", "spill_bytes", "smem_bytes", "repeats", "iters", "ms_median", "ms_min", "ms_mean", "ms_stdev",
              "tflops", "status"]


# ----------------------------------------------------------------------------- resources (CPU)
def parse_resources(report: str) -> dict:
    """``build.resource_report()`` text -> {(variant, op, out_dtype): {"regs", "spill_bytes", "stack"}}.

    The kernel's template arguments <CG, TN, TK, STAGES, EPI_WARPS, OP, OUT, NBUF> are read back from the
    mangled name (``...ILi2ELi256ELi128ELi5ELi8ELi1ELi0ELi1EE...``)."""
    out = {}
    for line in report.splitlines():
        m = re.match(r"variant_(\d+): (\S+) regs=(\d+) stack=(\d+) spill_stores=(\d+) spill_loads=(\d+)", line)
        if not m:
            continue
        args = [int(x) for x in re.findall(r"Li(\d+)E", m.group(2))]
        if len(args) < 8:
            continue
        out[(int(m.group(1)), args[5], args[6])] = {"regs": int(m.group(3)), "stack": int(m.group(4)),
                                                    "spill_bytes": int(m.group(5)) + int(m.group(6))}
    return out


def prune(variants: list[dict], op: int, resources: dict | None = None, out_dtype: int = 0) -> list[dict]:
    """Drops the variants that cannot or should not run a layer: one staging buffer serves FC1 only (the
    residual needs a second one to land in), more than 227 KiB of shared memory, spilling kernels."""
    keep = []
    for v in variants:
        if op != OPS["fc1"] and v["staging_buffers"] < 2:
            continue
        if v.get("smem_bytes", 0) > 232448:
            continue
        r = (resources or {}).get((v["variant_id"], op, out_dtype))
        if r is not None and r["spill_bytes"] > 0:
            continue
        keep.append(v)
    return keep


# ----------------------------------------------------------------------------- table (CPU)
def beats(a: dict, b: dict, margin: float) -> bool:
    """Whether `a` is faster than `b` by more than `margin` and by more than the two deviations that the sweep recorded."""
    spread = sum(float(r.get("ms_stdev") or 0.0) for r in (a, b))
    return float(b["ms_median"]) - float(a["ms_median"]) > max(margin * float(a["ms_median"]), spread)


def best_rows(rows: list[dict], keep_margin: float = 0.02) -> list[dict]:
    """CSV rows -> dispatch rows {op, N, K, m_min, variant}.

    Per (op, N, K) the M ladder is walked upwards; the winner of the previous (smaller) M is kept unless
    another variant beats it by more than ``keep_margin`` and by more than the two deviations recorded (noise must not flip the
    table), and neighbouring M with the same winner collapse into one row whose ``m_min`` is the smallest of them (0 for the first).  At the
    smallest M a single-CTA variant within 3 % of the best is taken: a CTA pair waits for two free SMs side by side."""
    groups: dict[tuple, dict[int, list[dict]]] = {}
    for r in rows:
        if r["status"] != "ok":
            continue
        groups.setdefault((int(r["op"]), int(r["N"]), int(r["K"])), {}).setdefault(int(r["M"]), []).append(r)
    table = []
    for (op, n, k), by_m in sorted(groups.items()):
        prev = None
        for i, m in enumerate(sorted(by_m)):
            cands = sorted(by_m[m], key=lambda r: float(r["ms_median"]))
            best = cands[0]
            choice = int(best["variant"])
            if prev is None:
                choice = next((int(r["variant"]) for r in cands if str(r.get("cta_group")) == "1"
                               and float(r["ms_median"]) <= float(best["ms_median"]) * 1.03), choice)
            if prev is not None and prev != choice:
                mine = next((r for r in cands if int(r["variant"]) == prev), None)
                if mine is not None and not beats(best, mine, keep_margin):
                    choice = prev
            if choice != prev:
                table.append({"op": op, "N": n, "K": k, "m_min": 0 if i == 0 else m, "variant": choice})
            prev = choice
    return table


def emit_header(table: list[dict], source: str, path: Path = TABLE_HEADER) -> str:
    lines = ["// sl8_dispatch_table.h -- GENERATED by `python -m siglip_b200.sweep --emit-table " + source + "`.",
             "// One row per (layer, N, K, smallest M) -> kernel variant, from the sweep on B200; pick_variant() takes the",
             "// row with the largest m_min <= M for an exact (layer, N, K) match and asks its cost model otherwise.",
             "#pragma once", "",
             "struct Sl8DispatchRow { int op; int n; int k; long long m_min; int variant; };", "",
             "static const Sl8DispatchRow kSl8DispatchTable[] = {"]
    for r in table:
        lines.append(f"    {{{OP_ENUM[r['op']]}, {r['N']}, {r['K']}, {r['m_min']}LL, {r['variant']}}},")
    if not table:
        lines.append("    {-1, 0, 0, 0LL, 0},")
    lines += ["};", f"static const int kSl8DispatchRows = {max(len(table), 0)};", ""]
    text = "\n".join(lines)
    path.write_text(text)
    return text


def read_csv(path: Path) -> list[dict]:
    with open(path, newline="") as f:
        return list(csv.DictReader(f))


# ----------------------------------------------------------------------------- timing (GPU)
def ladder(per_image: int, octaves: int, per_octave: int) -> list[int]:
    """per_image * 2^j; where the last round of tiles weighs, also the points that divide an octave: into per_octave below 16 images,
    into half as many up to 46 656 rows."""
    points = []
    for j in range(octaves):
        m = per_image << j
        parts = 1 if j == octaves - 1 else per_octave if j < 4 else max(1, per_octave // 2) if m < 46656 else 1
        points += [m + m * q // parts for q in range(parts)]
    return points


def capture(go, iters: int, stream):
    """A graph of `iters` launches."""
    import torch
    with torch.cuda.stream(stream):
        go()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        for _ in range(iters):
            go()
    return graph


def replay_ms(graph, iters: int, lead: int = 0, count: int = 1) -> float:
    """Milliseconds per launch over `count` replays of a graph of `iters` launches, `lead` untimed ones directly ahead of them."""
    import torch
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for _ in range(lead):
        graph.replay()
    e0.record()
    for _ in range(count):
        graph.replay()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / (iters * count)


# From this many rows on the board's power limit sets the pace, and a sample is 100 ms of a variant's own launches behind 100 ms of the
# same: bursts of ten launches, paced by what ran ahead of them, differ by 1 - 9 % from one another and 25 ms by 1 - 6 %, 100 ms by 0.2 -
# 0.7 % (FC2 1 152 x 4 304 at 46 656 and 373 248 rows, patch embedding 1 152 x 588 at 186 624, FC1 4 304 x 1 152 at 46 656, twenty samples each).
SUSTAINED_FROM = 10_000
SUSTAINED_MS = 100.0


def run_sweep(shape_sets: list[str], m_steps: int, repeats: int, iters: int, out_path: Path, variants_only=None,
              max_rows: int | None = None, log=print, per_octave: int = 1) -> list[dict]:
    """Times every admissible variant on every (layer, N, K) of the named shape sets over the M ladder."""
    import torch
    import siglip_b200
    from siglip_b200 import build, layers, synth
    from siglip_b200.lib import SL8Error

    dev = "cuda"
    eng = siglip_b200.Engine(0)
    stream = torch.cuda.Stream()
    resources = parse_resources(build.resource_report())
    all_variants = [layers.describe_variant(v) for v in range(layers.num_variants())]
    rows = []
    out_path.parent.mkdir(parents=True, exist_ok=True)
    with open(out_path, "w", newline="") as f:
        w = csv.DictWriter(f, fieldnames=CSV_FIELDS)
        w.writeheader()
        for set_name in shape_sets:
            for op_name, n, k, per_image in SHAPE_SETS[set_name]:
                op = OPS[op_name]
                for m in ladder(per_image, m_steps, per_octave):
                    if max_rows is not None and m > max_rows:
                        break
                    if op == 0:
                        p = synth.make_patch_embed(m, n, k, per_image, seed=0, device=dev, pixels=True)
                    elif op == 1:
                        p = synth.make_fc1(m, n, k, seed=0, device=dev)
                    else:
                        p = synth.make_fc2(m, n, k, seed=0, device=dev)
                    sa = torch.tensor([p.scale_a], device=dev)
                    sb = torch.tensor([p.scale_b], device=dev)
                    # Three operand sets taken in turn, so that no launch finds its A rows or its output lines in L2
                    # (the protocol of bench.py); weights, bias and table stay, as they would in a model.
                    sets = 3

                    def clone_pitched(t):
                        return torch.empty_strided(t.shape, t.stride(), dtype=t.dtype, device=t.device).copy_(t)

                    a_sets = [p.A] + [clone_pitched(p.A) for _ in range(sets - 1)]
                    d_sets = [torch.empty((m, n), dtype=torch.bfloat16, device=dev) for _ in range(sets)]
                    r_sets = [p.residual] + [p.residual.clone() for _ in range(sets - 1)] if op == 2 else None
                    tbl = eng.padded_table(p.table) if p.table is not None else None
                    turn = [0]

                    def go():
                        i = turn[0] % sets
                        turn[0] += 1
                        if op == 1:
                            eng.fc1_gelu(a_sets[i], p.B, p.bias, scale_a=sa, scale_b=sb, out=d_sets[i])
                        elif op == 2:
                            eng.fc2_residual(a_sets[i], p.B, p.bias, r_sets[i], scale_a=sa, scale_b=sb, out=d_sets[i])
                        else:
                            eng.patch_embed(a_sets[i], p.B, tbl, period=p.period, scale_a=sa, scale_b=sb, out=d_sets[i])

                    # Variants are timed in rounds (every variant once per round), not one after the other: the chip is
                    # power-bound under these kernels and whoever runs last on a warm GPU would look slower.
                    cands = [v for v in prune(all_variants, op, resources)
                             if variants_only is None or v["variant_id"] in variants_only]
                    sustained = m >= SUSTAINED_FROM
                    order = random.Random(m)
                    samples = {v["variant_id"]: [] for v in cands}
                    status = {v["variant_id"]: "ok" for v in cands}
                    graphs, count = {}, {}
                    for rnd in range(repeats + 1):                 # round 0 captures and warms up and is not recorded
                        for v in order.sample(cands, len(cands)):
                            vid = v["variant_id"]
                            if status[vid] != "ok":
                                continue
                            try:
                                if rnd == 0:
                                    eng.set_variant(vid)
                                    graphs[vid] = capture(go, iters, stream)
                                ms = replay_ms(graphs[vid], iters, *((count[vid], count[vid]) if rnd and sustained else ()))
                                eng.device_status()
                                if rnd:
                                    samples[vid].append(ms)
                                else:
                                    count[vid] = math.ceil(SUSTAINED_MS / (ms * iters))
                            except SL8Error as e:        # a bounded device wait ran out, or the variant refused the shape
                                status[vid] = "timeout" if "TIMEOUT" in str(e).upper() else "error"
                    del graphs
                    for v in cands:
                        vid = v["variant_id"]
                        res = resources.get((vid, op, 0), {})
                        row = {"op": op, "M": m, "N": n, "K": k, "variant": vid, "cta_group": v["cta_group"],
                               "tile_n": v["tile_n"], "tile_k": v["tile_k"], "stages": v["stages"],
                               "epi_warps": v["epi_warps"], "staging_buffers": v["staging_buffers"],
                               "regs": res.get("regs", ""), "spill_bytes": res.get("spill_bytes", ""),
                               "smem_bytes": v.get("smem_bytes", ""), "repeats": repeats, "iters": iters}
                        ms = samples[vid]
                        if status[vid] == "ok" and ms:
                            row.update(ms_median=statistics.median(ms), ms_min=min(ms), ms_mean=statistics.fmean(ms),
                                       ms_stdev=statistics.pstdev(ms), tflops=p.flops() / statistics.median(ms) / 1e9,
                                       status="ok")
                        else:
                            row.update(ms_median="", ms_min="", ms_mean="", ms_stdev="", tflops="",
                                       status=status[vid] if status[vid] != "ok" else "error")
                        w.writerow(row)
                        f.flush()
                        rows.append({k2: str(v2) for k2, v2 in row.items()})
                    ok = [r for r in rows if r["op"] == str(op) and r["M"] == str(m) and r["N"] == str(n) and r["status"] == "ok"]
                    if ok:
                        b = min(ok, key=lambda r: float(r["ms_median"]))
                        log(f"{op_name} M={m} N={n} K={k}: best v{b['variant']} {float(b['ms_median']) * 1e3:.1f} us "
                            f"{float(b['tflops']):.0f} TFLOP/s  ({len(ok)} variants)")
                    del p, a_sets, d_sets, r_sets
                    torch.cuda.empty_cache()
    eng.set_variant(-1)
    return rows


# ----------------------------------------------------------------------------- the cost model of pick_variant
# (class, N, K): the widths of the two encoders and of no model's, down to a single narrow tile, per kind of epilogue the model knows.
NARROW = [(400, 592), (320, 1280), (256, 4176), (144, 1616), (64, 592), (16, 80)]
MODEL_SHAPES = {
    "GELU": [(4304, 1152), (3072, 768), (1600, 512), (4800, 1600), (1152, 4304), (1600, 4800)] + NARROW,
    "TANH": [(4304, 1152), (3072, 768), (1152, 4304), (1600, 4800)] + NARROW,
    "NONE": [(3456, 1152), (2304, 768), (4800, 1600), (1536, 512), (1152, 4304), (1600, 4800)] + NARROW,
    "FC2": [(1152, 4304), (768, 3072), (1152, 1152), (768, 768), (1600, 4800), (512, 1600), (384, 1536), (272, 2128)] + NARROW,
    "PE": [(1152, 588), (768, 768), (1600, 768), (640, 588), (384, 768), (272, 588)] + [(n, k) for n, k in NARROW if k < 2048],
}
MODEL_ROWS = [50, 128, 196, 256, 392, 512, 729, 1000, 1200, 1458, 1568, 1800, 2048, 2400, 2916, 3300, 3700, 4374, 5003, 5400, 5832, 6400, 7000,
              7800, 8748, 9500, 10300, 11664, 13000, 14580, 16000, 17496, 20000, 23328, 27000, 32000, 39000, 46656, 93312, 186624]
MODEL_CSV = PKG / "sweeps" / "b200_model.csv"
MODEL_HEADER = PKG / "csrc" / "sl8_cost_model.h"


def shown_path(path: Path) -> str:
    try:
        return str(path.resolve().relative_to(PKG.parent))
    except ValueError:
        return str(path)


def variant_tiles() -> dict:
    """{variant: (CTAs per tile, tile N)} from the list they are compiled from."""
    return {int(v): (int(cg), int(tn)) for v, cg, tn in re.findall(r"X\((\d+), (\d), (\d+),", (PKG / "csrc" / "sl8_variants.h").read_text())}


def cost_constants(path: Path = MODEL_HEADER) -> dict:
    """{(class, variant): (start, first, next, tile)} as the committed header holds them."""
    found = re.findall(r"\{COST_(\w+), (\d+), ([\d.]+)f, ([\d.]+)f, ([\d.]+)f, ([\d.]+)f\}", path.read_text())
    return {(c, int(v)): tuple(map(float, k)) for c, v, *k in found}


def emit_model(constants: dict, source: str, path: Path = MODEL_HEADER) -> None:
    lines = ["// sl8_cost_model.h -- GENERATED by `python -m siglip_b200.sweep --fit-model " + source + "`: class of epilogue, variant, start, first, next, tile."]
    for (cls, v), k in constants.items():
        lines.append(f"    {{COST_{cls}, {v}, " + ", ".join(f"{x!r}f" for x in k) + "},")
    path.write_text("\n".join(lines) + "\n")


def model_us(k: tuple, cg: int, tn: int, M: int, N: int, K: int, sms: int = 148) -> float:
    """The formula beside kVariantCost."""
    tiles, k_blocks = -(-M // (128 * cg)) * -(-N // tn), -(-K // 128)
    rounds = -(-tiles // (sms // cg))
    return k[0] + k_blocks * k[1] + (rounds - 1) * max(k_blocks * k[2], k[3])


def cheapest(cls: str, M: int, N: int, K: int, clusters: int | None = None) -> int:
    """The variant that the committed constants pick, on a handle held to `clusters` CTAs or pairs or on the whole chip."""
    tiles = variant_tiles()
    us = lambda v, k: model_us(k, *tiles[v], M, N, K, sms=min(148 // tiles[v][0], clusters or 148) * tiles[v][0])
    return min((us(v, k), v) for (c, v), k in cost_constants().items() if c == cls)[1]


def asked_rows(rows: list[dict]) -> list[dict]:
    """The points of the sweep that the dispatch table leaves to the model (of a class that the table has whole: all of them)."""
    table = {(r["op"], r["N"], r["K"]) for r in best_rows(read_csv(PKG / "sweeps" / "b200.csv"))}
    ops = {"GELU": OPS["fc1"], "FC2": OPS["fc2"], "PE": OPS["pe"]}
    asked = [r for r in rows if (ops.get(r["cls"]), int(r["N"]), int(r["K"])) not in table]
    return asked + [r for r in rows if r["cls"] not in {a["cls"] for a in asked}]


def model_regret(rows: list[dict], constants: dict, variants: dict) -> dict:
    """{class: [(how much longer than the fastest variant the cheapest one by the formula took, the row)]}."""
    out = {}
    for r in rows:
        m, n, k = int(r["M"]), int(r["N"]), int(r["K"])
        times = {int(f[1:]): float(t) for f, t in r.items() if f[0] == "v" and t}
        mine = [(model_us(c, *variants[v], m, n, k), v) for (cls, v), c in constants.items() if cls == r["cls"] and v in times]
        out.setdefault(r["cls"], []).append((times[min(mine)[1]] / min(times.values()) - 1.0, r))
    return out


def fit_model(rows: list[dict], constants: dict, variants: dict, steps=(0.98, 1.02, 0.95, 1.05, 0.9, 1.1), least: float = 2e-4) -> dict:
    """`constants` with every number moved in small steps, one after the other and as long as it helps, to where the variant
    picked is slower than the fastest by less: on average plus a tenth of the worst case, from 512 columns on and below added up (the
    worst cases are narrow, and would hide the others').  A step has to gain `least`: smaller ones follow the noise of one sweep.  Its own
    result it leaves as it is."""
    out = dict(constants)
    for cls in sorted({c for c, _ in constants}):
        mine = [v for c, v in constants if c == cls]
        points = [(int(r["M"]), int(r["N"]), int(r["K"]), {int(f[1:]): float(t) for f, t in r.items() if f[0] == "v" and t}) for r in rows if r["cls"] == cls]
        points = [(m, n, k, {v: t[v] / min(t.values()) - 1.0 for v in mine if v in t}) for m, n, k, t in points]
        cost = {v: [model_us(out[cls, v], *variants[v], m, n, k) for m, n, k, _ in points] for v in mine}

        def lost():
            return [t[min((cost[v][i], v) for v in t)[1]] for i, (_, _, _, t) in enumerate(points)]

        halves = [h for h in ([i for i, p in enumerate(points) if p[1] >= 512], [i for i, p in enumerate(points) if p[1] < 512]) if h]

        def score(now):
            return sum(statistics.fmean(now[i] for i in h) + 0.1 * max(now[i] for i in h) for h in halves)

        best, moved = score(lost()), True
        while moved:
            moved = False
            for v in mine:
                for j in range(4):
                    for f in steps:
                        old, kept = out[cls, v], cost[v]
                        out[cls, v] = old[:j] + (float(f"{old[j] * f:.3g}"),) + old[j + 1:]
                        cost[v] = [model_us(out[cls, v], *variants[v], m, n, k) for m, n, k, _ in points]
                        now = score(lost())
                        if now < best - least:
                            best, moved = now, True
                        else:
                            out[cls, v], cost[v] = old, kept
    return out


def run_model_sweep(out_path: Path, repeats: int = 3, log=print) -> None:
    """Graph-replay microseconds of every admissible variant over MODEL_SHAPES x MODEL_ROWS, two operand sets in turn."""
    import torch
    import siglip_b200
    from siglip_b200 import build, layers, lib, synth

    eng, stream = siglip_b200.Engine(0), torch.cuda.Stream()
    resources = parse_resources(build.resource_report())
    every = [layers.describe_variant(v) for v in range(layers.num_variants())]
    gen = torch.Generator(device="cuda").manual_seed(0)
    normal = lambda *s: torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16)
    codes = lambda r, c: (torch.randint(0, 256, (r, synth.pitch128(c)), generator=gen, device="cuda", dtype=torch.uint8) & 0xBF)[:, :c]
    s = torch.full((1,), 0.01, device="cuda")
    with open(out_path, "w", newline="") as f:
        w = csv.writer(f)
        w.writerow(["cls", "N", "K", "M"] + [f"v{v['variant_id']}" for v in every])
        for cls, shapes in MODEL_SHAPES.items():
            op = OPS["pe"] if cls == "PE" else OPS["fc2"] if cls == "FC2" else OPS["fc1"]
            for n, k in shapes:
                B, bias, table = codes(n, k), normal(n), normal(729 + 128, n)
                for m in MODEL_ROWS:
                    if m > 46656 and (op, n, k) not in [(OPS[x[0]], x[1], x[2]) for shape_set in SHAPE_SETS.values() for x in shape_set]:
                        break
                    A, D = [codes(m, k) for _ in range(2)], [torch.empty((m, n), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
                    res = [normal(m, n) for _ in range(2)] if cls == "FC2" else None
                    turn = [0]

                    def go():
                        i = turn[0] = 1 - turn[0]
                        kw = dict(scale_a=s, scale_b=s, out=D[i])
                        if cls == "PE":
                            eng.patch_embed(A[i], B, table, period=729, **kw)
                        elif cls == "FC2":
                            eng.fc2_residual(A[i], B, bias, res[i], **kw)
                        elif cls == "NONE":
                            eng.linear_bias(A[i], B, bias, **kw)
                        else:
                            eng.fc1_gelu(A[i], B, bias, flags=lib.SL8_FLAG_GELU_HW_TANH if cls == "TANH" else 0, **kw)

                    iters, us = 12 if m <= 8748 else 6, {}
                    for v in prune(every, op, resources):
                        eng.set_variant(v["variant_id"])
                        try:
                            graph = capture(go, iters, stream)
                            replay_ms(graph, iters)
                            us[v["variant_id"]] = statistics.median(replay_ms(graph, iters) for _ in range(repeats)) * 1e3
                        except lib.SL8Error:
                            pass
                    eng.set_variant(-1)
                    eng.device_status()
                    w.writerow([cls, n, k, m] + [f"{us[v['variant_id']]:.3f}" if v["variant_id"] in us else "" for v in every])
                    f.flush()
                    del A, D, res
                log(f"{cls} {n} x {k}")


def main(argv=None) -> int:
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("--shapes", default="so400m,b16", help="comma-separated shape sets: " + ", ".join(SHAPE_SETS))
    ap.add_argument("--m-steps", type=int, default=11, help="M from rows_per_image to rows_per_image * 2^(m-steps - 1)")
    ap.add_argument("--per-octave", type=int, default=8, help="points of the M ladder per doubling, up to 16 images; half as many up to 46 656 rows")
    ap.add_argument("--max-rows", type=int, default=None)
    ap.add_argument("--repeats", type=int, default=5)
    ap.add_argument("--iters", type=int, default=10)
    ap.add_argument("--out", type=Path, default=PKG / "sweeps" / "b200.csv")
    ap.add_argument("--variants", default="", help="restrict to these variant ids")
    ap.add_argument("--emit-table", type=Path, default=None, metavar="CSV",
                    help="no GPU work: turn this CSV into csrc/sl8_dispatch_table.h")
    ap.add_argument("--model-sweep", action="store_true", help="time the points of the cost model into " + MODEL_CSV.name)
    ap.add_argument("--fit-model", type=Path, default=None, metavar="CSV",
                    help="no GPU work: move the constants of csrc/sl8_cost_model.h to where they pick best on this CSV")
    a = ap.parse_args(argv)
    if a.model_sweep:
        run_model_sweep(MODEL_CSV)
        return 0
    if a.fit_model is not None:
        variants, constants = variant_tiles(), cost_constants()
        rows = asked_rows(read_csv(a.fit_model))
        fitted = fit_model(rows, constants, variants)
        emit_model(fitted, shown_path(a.fit_model))
        for name, k in (("before", constants), ("after", fitted)):
            for cls, lost in model_regret(rows, k, variants).items():
                print(f"{name} {cls}: {100 * statistics.fmean(x for x, _ in lost):.2f} % off the fastest on average, {100 * max(x for x, _ in lost):.1f} % at worst")
        return 0
    if a.emit_table is not None:
        table = best_rows(read_csv(a.emit_table))
        emit_header(table, shown_path(a.emit_table))
        print(f"{len(table)} rows -> {TABLE_HEADER}")
        return 0
    only = {int(x) for x in a.variants.split(",")} if a.variants else None
    run_sweep(a.shapes.split(","), a.m_steps, a.repeats, a.iters, a.out, only, a.max_rows, per_octave=a.per_octave)
    print(f"wrote {a.out}")
    return 0


if __name__ == "__main__":
    sys.exit(main())
