"""Autotuner of the GB300 FFT backend.

For each grid shape it measures, on the GPU at hand, the choices an engine
can make and writes the fastest into the tuning cache that engines read at
creation (tune_cache.txt beside this file, or $GBFFT_TUNE_CACHE):

  * the radix plan of power-of-two axes: 16 or 8 or 4 points a thread on lines
    of at most 256 points (8) or 128 (4); of axes of 512 or 1024 points: 16 points per thread
    (radix 16 stages) or 32 (two radix-32 stages); of axes of 243, 270,
    360, 384, 400 points: the balanced plan or the two-stage one (2)
                                                               -> e_x, e_y, e_z
  * row layout: padded work-area rows, flat z passes          -> pad, flat
  * strided passes staged by bulk tensor copies or one-shot    -> tma
  * the tile shape (lines per CTA) of every pass kind          -> r2c, c2r,
                                                                  c2c_x, c2c_y,
                                                                  c2c_z, xy_fused
  * launch form of the one-shot kernels: one CTA per tile, or clusters of
    2, 4 or 8 neighbouring CTAs (with or without a start barrier)
                                                               -> cl_<pass>,
                                                                  cls_<pass>
  * pass fusion: x and y passes of each z-plane in one kernel  -> fuse

Plans, layouts and the staging choice interact (the bulk-copy kernel needs
rows a tensor map can describe, and shares the axis plan's twiddles), so
every combination of the three is timed first; tile shapes and launch forms
are then tuned pass by pass for the fastest.  The measured step is the
benchmark's: one r2c then one c2r, per-pass device times from CUDA events on
the launching stream.

    python tune.py [--out FILE] [--shapes prec,fmt,nx,ny,nz ...]
"""
import argparse
import itertools
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
if HERE not in sys.path:
    sys.path.insert(0, HERE)

import gbfft  # noqa: E402

# prec format nx ny nz: the benchmark's grids
DEFAULT_SHAPES = [
    (4, 1, 1024, 1024, 512), (4, 3, 1024, 1024, 512),
    (4, 1, 384, 400, 243), (8, 1, 384, 400, 243),
    (4, 1, 360, 270, 210), (8, 1, 360, 270, 210),
    (4, 1, 256, 256, 256), (8, 1, 64, 64, 64),
    # reduced grids of the 1024 x 1024 x 512 passes, for profiling
    (4, 1, 1024, 1024, 128), (4, 1, 512, 256, 512),
]
TILES = [1, 2, 4, 8, 16, 32]
MARGIN = 0.99
# launch forms of the one-shot kernels: (cluster CTAs, start barrier)
LAUNCHES = [(0, 0), (2, 0), (2, 1), (4, 1), (8, 1)]
LAYOUTS = [(0, True), (1, True), (2, True), (0, False), (1, False)]


def measure(eng, x, s, y, steps=6, warm=2):
    """{pass: ms per launch} and the step time in ms."""
    import torch
    for _ in range(warm):
        eng.r2c(x, s)
        eng.c2r(s, y)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        eng.r2c(x, s)
        eng.c2r(s, y)
    e1.record()
    torch.cuda.synchronize()
    step = e0.elapsed_time(e1) / steps
    eng.set_profiling(True)
    for _ in range(steps):
        eng.r2c(x, s)
        eng.c2r(s, y)
    torch.cuda.synchronize()
    prof = eng.profile()
    eng.set_profiling(False)
    return {k: v[1] / v[0] for k, v in prof.items()}, step


BALANCED = {243: 9, 270: 30, 360: 30, 384: 24, 400: 20}  # points of the balanced plans


def plan_choices(prec, n):
    """Points a thread to try on an axis of n points ([None]: one plan).  In
    double precision lines of these lengths run in fixed point, with one plan
    each, whatever set_plan keeps."""
    if prec == 8:
        return [None]
    if n in (512, 1024):
        return [16, 32]
    if n in BALANCED:
        return [BALANCED[n], 2]
    if n in (16, 32, 64, 128):
        return [16, 8, 4]  # short lines: more threads on small grids
    return [16, 8] if n == 256 else [None]


def launch_choices(prec, kind, n, points):
    """Launch forms to try: clusters exist for the compile-time power-of-two
    kernels, which are single precision's."""
    return [(0, 0)] if prec == 8 or kind == "xy_fused" or not points or n & (n - 1) else LAUNCHES


def take_tile(eng, kind, lines):
    """Sets a tile; whether the pass runs it (a refused one, or one that the
    kernel in use replaces by the built-in tile, is not worth timing)."""
    try:
        eng.set_tile(kind, lines)
    except gbfft.GbfftError:
        return False
    return eng.tuning()["tiles"][kind] == lines


def tune_shape(prec, fmt, nx, ny, nz, log=print):
    import torch
    rdt = torch.float32 if prec == 4 else torch.float64
    eng = gbfft.Engine(fmt, nx, ny, nz, prec=prec)
    x = torch.randn((nz, ny, nx), dtype=rdt, device="cuda")
    s = eng.empty_spectral()
    y = eng.empty_physical()
    opts = {axis: plan_choices(prec, n) for axis, n in ((0, nx), (1, ny), (2, nz))}
    eng.set_fusion(False)

    def apply(ex, ey, ez, layout, tma):
        for axis, pts in ((0, ex), (1, ey), (2, ez)):
            if pts:
                eng.set_plan(axis, pts)
        eng.set_layout(*layout)
        eng.set_tma(tma)

    # 1. plan x layout x staging, built-in tiles: the fastest step
    best = None
    for ex, ey, ez in itertools.product(opts[0], opts[1], opts[2]):
        for layout in LAYOUTS:
            for tma in (True, False):
                apply(ex, ey, ez, layout, tma)
                _, st = measure(eng, x, s, y)
                log("  e_x=%s e_y=%s e_z=%s pad=%d flat=%d tma=%d: %.4f ms" % (
                    ex, ey, ez, layout[0], layout[1], tma, st))
                # the built-in layout and staging unless another wins by 1 %
                builtin = layout == LAYOUTS[0] and tma
                key = st if builtin else st / MARGIN
                if best is None or key < best[0]:
                    best = (key, ex, ey, ez, layout, tma)
    _, ex, ey, ez, layout, tma = best
    apply(ex, ey, ez, layout, tma)

    # 2. tile shape and launch form of every pass kind
    times, _ = measure(eng, x, s, y)
    pts = eng.tuning()["points"]
    tiles, clusters = {}, {}
    for kind, t0 in times.items():
        bt, bl, bc = t0, 0, (0, 0)
        axis = {"c2c_x": 0, "c2c_y": 1, "c2c_z": 2}.get(kind, 0 if fmt == 1 else 2)
        n = (nx, ny, nz)[axis]
        for clus in launch_choices(prec, kind, n, pts[axis]):
            eng.set_cluster(kind, *clus)
            for L in [0] + TILES:
                if not take_tile(eng, kind, L):
                    continue
                t = measure(eng, x, s, y, steps=4, warm=1)[0].get(kind, t0)
                # a choice other than the built-in one must win by 1 %
                if t < bt and t < t0 * MARGIN:
                    bt, bl, bc = t, L, clus
                eng.set_tile(kind, 0)
        eng.set_cluster(kind, 0, 0)
        tiles[kind] = bl
        clusters[kind] = bc
    for kind, L in tiles.items():
        if L:
            eng.set_tile(kind, L)
    for kind, c in clusters.items():
        if c[0]:
            eng.set_cluster(kind, *c)
    log("  tiles %s clusters %s" % (tiles, clusters))

    # 3. pass fusion
    _, step_plain = measure(eng, x, s, y)
    fuse = 0
    eng.set_fusion(True)
    times_f, step_fused = measure(eng, x, s, y)
    if "xy_fused" in times_f and step_fused < step_plain:
        fuse = 1
    log("  step %.4f ms unfused, %.4f ms fused%s" % (step_plain, step_fused,
                                                    "" if "xy_fused" in times_f else " (no fused kernel)"))
    eng.close()
    fields = ["%d %d %d %d %d" % (prec, fmt, nx, ny, nz), "fuse=%d" % fuse]
    if layout[0]:
        fields.append("pad=%d" % layout[0])
    if not layout[1]:
        fields.append("flat=0")
    if not tma:
        fields.append("tma=0")
    if ex:
        fields.append("e_x=%d" % ex)
    if ey:
        fields.append("e_y=%d" % ey)
    if ez:
        fields.append("e_z=%d" % ez)
    for kind, L in sorted(tiles.items()):
        if L:
            fields.append("%s=%d" % (kind, L))
    for kind, c in sorted(clusters.items()):
        if c[0]:
            fields.append("cl_%s=%d" % (kind, c[0]))
            if c[1]:
                fields.append("cls_%s=1" % kind)
    return " ".join(fields), min(step_plain, step_fused if fuse else step_plain)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--out", default=os.path.join(HERE, "tune_cache.txt"))
    ap.add_argument("--shapes", nargs="*", help="prec,fmt,nx,ny,nz")
    args = ap.parse_args()
    shapes = [tuple(int(v) for v in s.split(",")) for s in args.shapes] if args.shapes else DEFAULT_SHAPES
    gbfft.lib()
    gbfft.set_tune_cache("")  # measure from the built-in choices
    lines = ["# GB300 tuning cache written by tune.py: prec format nx ny nz key=value ...",
             "# keys: fuse, e_x/e_y/e_z (points per thread of the axis plans), lines per CTA per pass,",
             "# cl_<pass> / cls_<pass> (cluster launch: CTAs a cluster / start barrier), pad / flat",
             "# (row layout), tma (strided passes staged by bulk tensor copies; default 1)"]
    for shp in shapes:
        print("shape", shp, flush=True)
        line, ms = tune_shape(*shp)
        print("  ->", line, "(%.4f ms)" % ms, flush=True)
        lines.append(line)
    with open(args.out, "w") as f:
        f.write("\n".join(lines) + "\n")
    print("wrote", args.out)


if __name__ == "__main__":
    main()
