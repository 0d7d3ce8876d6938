"""Tile-shape autotuner of the multigrid smoother.

The levels above the one-block sub-cycle are smoothed by tiled kernels whose tile
edge is 16 or 32, or, where they are large and in double, swept in strips; the default
picks by the level's size.  Whether that is the faster choice depends on the level's
size, the operator and the precision, so ``tune_tile_edges`` measures it: for every
assignment of {16, 32}, and of the strips where they are a level's default, it times
one V-cycle on the context's current operator (``diva_profile_kernel`` kind 3, CUDA
events on the context's stream), keeps the fastest, and sets it with
``diva_set_tile_edges``.  The solution is the same bit for bit whatever the shape (every
smoother reproduces the per-colour sweeps), so tuning changes time only.  Results are
cached per grid shape and configuration in a JSON file when ``cache`` is given, so an
ensemble tunes each member size once.
"""
import itertools
import json
import os


def cache_key(ctx):
    """Grid and configuration, and which shapes the choice was between (``strips``)."""
    g, c = ctx.grid, ctx.cfg
    return f"{g.nx}x{g.ny}x{g.nz}:prec{int(c.precision)}:margin{int(c.choice_ice_margin)}:strips"


def candidates(edges, strips=()):
    """Every assignment of 16 / 32 to the tiled levels (edge != 0) of ``edges``, and of 0,
    the default, to those of them that it sweeps in strips (``strips`` != 0)."""
    tiled = [l for l, e in enumerate(edges) if e]
    options = [(0, 16, 32) if l < len(strips) and strips[l] else (16, 32) for l in tiled]
    for combo in itertools.product(*options):
        out = [0] * len(edges)
        for l, v in zip(tiled, combo):
            out[l] = v
        yield out


def tune_tile_edges(ctx, reps=20, trials=3, cache=None):
    """Pick and set the fastest shapes for ``ctx``; returns (edges, {candidate: ms}), the
    edges as ``get_tile_edges`` gives them then.  Contexts of other backends than the CUDA
    library have no tiles: ([], {})."""
    if getattr(getattr(ctx, "backend", None), "name", "cuda") != "cuda":
        return [], {}
    key = cache_key(ctx)
    if cache and os.path.exists(cache):
        with open(cache) as f:
            known = json.load(f)
        if key in known:
            ctx.set_tile_edges(known[key])
            return ctx.get_tile_edges(), {}
    ctx.nonlinear_residual()          # coefficients and operator at the current state
    ctx.set_tile_edges([])
    default = ctx.get_tile_edges()
    strips = ctx.get_strip_rows() if hasattr(ctx, "get_strip_rows") else ()
    timings = {}
    for e in candidates(default, strips):
        ctx.set_tile_edges(e)
        timings[tuple(e)] = min(ctx.profile_kernel(3, reps)[0] for _ in range(trials))
    best = list(min(timings, key=timings.get)) if timings else default
    ctx.set_tile_edges(best)
    if cache:
        known = {}
        if os.path.exists(cache):
            with open(cache) as f:
                known = json.load(f)
        known[key] = best
        with open(cache, "w") as f:
            json.dump(known, f, indent=1, sort_keys=True)
    return ctx.get_tile_edges(), timings
