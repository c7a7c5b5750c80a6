"""Compressed FSST rows with runs of 255s of chosen lengths (a 255 is an escape; the byte after it is literal, a 255 too)."""
import numpy as np

RUNS = (1, 2, 3, 4, 5, 7, 8, 62, 63, 64, 65, 66, 127, 128, 129, 200)


def run_row(rng, run, before, after):
    """`before` plain codes, a run of that many 255s, the literal of its last escape when it has one, `after` plain codes."""
    code = lambda k: bytes(rng.integers(0, 255, k, dtype=np.uint8))
    return code(before) + b"\xff" * run + code(run % 2) + code(after)


def rows(rng, kind):
    """1024 rows: `runs` of any length inside rows, `short` ones (below 64) alone, `cut` by row ends at random."""
    out = []
    for i in range(1024):
        if i % 9:
            out.append(bytes(rng.integers(0, 255, int(rng.integers(0, 9)), dtype=np.uint8)))
            continue
        run = int(rng.choice([r for r in RUNS if kind == "runs" or r < 64]))
        row = run_row(rng, run, int(rng.integers(0, 140)), int(rng.integers(1, 6)))
        if kind == "cut" and i % 27 == 0:
            row = row[: int(rng.integers(1, len(row) + 1))]
        out.append(row)
    return out
