"""The step kernels' tile order (groups of CTAs that take a run of tiles in turn) over grids and batches
of every proportion: one CTA, fewer CTAs than windows, more CTAs than tiles, groups that end inside
windows.  The fields are those of the default grid bit for bit, and every window's sums are those of its
own velocity field."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _specs(sizes):
    from particuology_hydraulic_penalty_b200 import windows as wgen
    from particuology_hydraulic_penalty_b200.batch import WindowSpec

    return [WindowSpec(n, wgen.make_window(n, "skeleton", 7 + k).particles, tau=0.7 + 0.05 * (k % 3),
                       force=(1e-6, 2e-6 * (k % 2), 0.0), subsamples=2 + k % 2) for k, n in enumerate(sizes)]


@pytest.mark.parametrize("precision,sizes", [
    ("fp32", [20]), ("fp32", [7, 9, 8]), ("fp32", [12] * 40 + [64] + [10] * 5), ("fp16", [48, 6, 64, 32]),
    ("fp64", [31, 18, 5]), ("fp64-exact", [17, 40, 6, 6, 22])])
def test_sums_and_fields_do_not_depend_on_the_grid(precision, sizes):
    from particuology_hydraulic_penalty_b200 import _native as nat
    from particuology_hydraulic_penalty_b200.batch import PscBatch

    ref = PscBatch(_specs(sizes), precision=precision, graph_steps=0)
    ref.run(6)
    fields = [ref.velocity_field(k) for k in range(ref.nwin)]
    pops = [w.f[ref.parity].clone() for w in ref.windows]
    grids = [0, 1, 5, 61, 296, 1000]
    for grid in grids:
        b = PscBatch(_specs(sizes), precision=precision, graph_steps=0, grid_ctas=grid)
        b.run(6)
        red = b.observe()
        for k in range(b.nwin):
            assert np.array_equal(b.windows[k].f[b.parity].cpu().numpy(), pops[k].cpu().numpy())
            for axis, slot in enumerate((nat.RED_UX, nat.RED_UY, nat.RED_UZ)):
                u = fields[k][1 + axis]
                # a sum of n terms in any order: at most n roundings of half an ulp of the absolute sum
                assert abs(red[k, slot] - u.sum()) <= u.size * 2.0 ** -53 * np.abs(u).sum()
            solid = b.geoms[k].solid.cpu().numpy()
            assert abs(red[k, nat.RED_SOLID] - solid.sum()) <= 1e-6 * max(1.0, solid.sum())
