"""Several series in one engine, grouped side by side: one, two, as many as
there are streams, one more and many, in 3D and 2D, replayed from graphs or
not, over several runs and the end. Per series the oracle's grouping of its
own frames."""

import numpy as np
import pytest

from conftest import same_spots
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("nseries,two_d", [(1, False), (2, False), (4, False), (5, True),
                                           (5, False), (9, False)])
def test_series_side_by_side(gpu_lib, nseries, two_d, graph):
    from dials_metal_spotfinder_b200.engine import Engine
    rng = np.random.default_rng(nseries)
    per_run, runs = 2, 4
    shapes = [(100 + 13 * k, 240 + 7 * k) for k in range(nseries)]
    frames = {}
    for k, (h, w) in enumerate(shapes):
        y, x = rng.integers(4, h - 4, 60), rng.integers(4, w - 4, 60)
        for z in range(per_run * runs):
            img = rng.poisson(0.5, (h, w)).astype(np.uint16)
            for j, (a, b) in enumerate(zip(y, x)):
                if (z + j) % 5 < 2:  # every reflection on two frames of five
                    img[a - 1:a + 2, b - 1:b + 2] += np.uint16(300)
            frames[k, z] = img
    got = [[] for _ in shapes]
    pixels = [[] for _ in shapes]
    with Engine(shapes * per_run, slots=2) as eng:
        eng.enable_grouping(two_d=two_d)
        eng.use_graph(graph)

        def collect():
            for k in range(nseries):
                got[k].append(eng.spots(k))
                pixels[k].append(eng.pixels(k))

        for r in range(runs):
            for f in range(per_run):
                for k in range(nseries):
                    eng.upload(r & 1, f * nseries + k, frames[k, r * per_run + f])
            eng.run(r & 1)
            collect()
        eng.finish()
        collect()
        counts = [eng.group_counts(k)[0] for k in range(nseries)]
    for k, (h, w) in enumerate(shapes):
        signals = [O.dext(frames[k, z])[1] for z in range(per_run * runs)]
        want = O.group(signals, h, w, two_d=two_d)
        assert counts[k] == want.counts, k
        same_spots(np.concatenate(got[k]), want.spots)
        assert np.concatenate(pixels[k]).tobytes() == want.pixels.tobytes(), k
