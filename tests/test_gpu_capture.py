"""A captured cf_step_adaptive replayed after a clone into the captured film:
the graph steps whatever state, params and settings the film then holds."""
import numpy as np
import pytest

import pyoracle as po
from canvaz_film import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tilts", [(0.0, 60.0), (60.0, 0.0), (0.0, 0.0)])
@pytest.mark.parametrize("w,h", [(96, 80), (208, 240)])  # few tiles, and more than a device has SMs
def test_a_captured_step_follows_a_clone(w, h, tilts):
    import torch

    import __graft_entry__ as g
    g.build()
    from canvaz_film.film import Film

    def film(tilt, seed):
        cv = synth.drip_canvas(w, h, seed, n_lines=12, per_cell_n=True, tilt_deg=tilt)
        f = Film(po.make_settings(cv.settings), w, h, capi.CF_PREC_FP32)
        f.set_tables(cv.pigtab, cv.cmf)
        f.write_state(cv.planes)
        for _ in range(2):
            f.step_adaptive(1e-3)
        f.sync()
        return f

    a, b = film(tilts[0], 3), film(tilts[1], 4)
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        for _ in range(2):  # back to the generation it starts from
            a.step_adaptive(1e-3, torch.cuda.current_stream().cuda_stream)
    a.clone_from(b)
    torch.cuda.synchronize()
    for _ in range(3):
        graph.replay()
        for _ in range(2):
            b.step_adaptive(1e-3)
    torch.cuda.synchronize()
    for p in ("h", "tmp", "flux", "strata_h", "color"):
        assert np.array_equal(a.plane(p), b.plane(p), equal_nan=True), p
