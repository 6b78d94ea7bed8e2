"""A dispatch run on its own leaves no tile still: the frame after it writes
every plane as a frame that leaves no tile out."""
import numpy as np
import pytest

import pyoracle as po
from canvaz_film import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", ["strata_pass", "laplacian"])
def test_a_frame_after_a_single_dispatch_leaves_no_tile_out(kernel):
    import __graft_entry__ as g
    g.build()
    from canvaz_film.film import Film
    cv = synth.drip_canvas(208, 160, 3, n_lines=2, per_cell_n=False)
    cv.settings.update(all_active=0)
    f = Film(po.make_settings(cv.settings), cv.w, cv.h, capi.CF_PREC_FP32)
    f.set_tables(cv.pigtab, cv.cmf)
    f.write_state(cv.planes)
    for _ in range(6):  # until the tiles far from the paint sleep
        f.update_params(2e-3, 1)
        f.encode_frame(1)
        f.sync()
    f.set_plane("h_next", np.full(f.n, 7.0))  # a frame copies h there in an inactive tile
    for _ in range(3):  # dry, dry twice over, still
        f.run(kernel)
    f.update_params(2e-3, 1)
    f.encode_frame(1)
    f.sync()
    assert (f.plane("h_next") == 7.0).sum() == 0
