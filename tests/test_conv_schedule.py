"""The convolution kernel's waits on barrier phases, on a model of its schedule.

A parity wait on phase p of a barrier is sound only if phase p - 1 is known to
be complete: otherwise it returns at once.  The model takes the ring lengths
from the kernel's source, deals the rows of a CTA's items to the epilogue
groups and the two MMA issuers as the kernel does, and derives what each
waiting thread knows (rows of a group and MMAs of an issuer complete in order;
a tile is overwritten after all its readers are done).  Needs no GPU."""
import itertools
import pathlib
import re

import pytest

SRC = pathlib.Path(__file__).parents[1] / "phasefield_coarsening_gb300" / "csrc" / "ppf_nn_conv.cu"


def constants():
    text = SRC.read_text()
    ring = re.search(r"int RING = ([^;]*);", text).group(1)
    return [int(v) for v in re.findall(r"(?<!== )\b\d+\b", ring)], int(re.search(r"int ND = (\d+);", text).group(1))


def items_of(ny, nyc):
    return [(k + 1) * ny // nyc - k * ny // nyc for k in range(nyc)]


def unsound(ns, groups, ring, nd):
    rows, readers, tiles = [], {}, 0
    for n in ns:
        for i in range(n):
            rows.append(tiles + i + 1)
            for t in range(tiles + i, tiles + i + 3):
                readers.setdefault(t, set()).add(len(rows) - 1)
        tiles += n + 2

    def known(done, complete):
        done, complete, size = set(done), set(complete), -1
        while size != len(done) + len(complete):
            size = len(done) + len(complete)
            done |= {r - groups for r in done if r >= groups}
            complete |= {rows[r] + d for r in done for d in (-1, 0, 1)} | {t - 2 for t in complete if t >= 2}
            done |= {r for t in complete if t >= nd for r in readers[t - nd]}
        return done, complete

    for r, qy in enumerate(rows):                   # an epilogue group waits for its row's three tiles
        seen = known({r - groups} if r >= groups else (), ())
        for t in (qy - 1, qy, qy + 1):
            if t >= nd and t - nd not in seen[1]:
                yield "tile", r, t
            seen = known(seen[0], seen[1] | {t})
    for q in range(tiles):                          # an issuer waits for row q's data and for its tile
        done, complete = known({r for u in range(q - 2, -1, -2) if u >= nd for r in readers[u - nd]}, ())
        if q >= 2 * nd and not readers[q - 2 * nd] <= done:
            yield "release", q
        if q >= ring and ring % 2 and q - ring not in complete:
            yield "data", q


@pytest.mark.parametrize("groups", [2, 3])
def test_every_wait_knows_the_phase_before(groups):
    rings, nd = constants()
    shapes = [tuple(items_of(ny, nyc)[:8]) for ny in range(2, 13) for nyc in range(1, ny // 2 + 1)]
    shapes += [(n,) * 8 for n in range(2, 8)] + list(itertools.product(range(2, 4), repeat=5))
    assert min(min(s) for s in shapes) == 2
    for ring in rings:
        for ns in shapes:
            assert not list(unsound(ns, groups, ring, nd)), (ring, ns)
