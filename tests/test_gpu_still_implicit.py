"""Still tiles and the implicit solve's own leaving out (tiles without paint):
every plane of a film whose frames take implicit steps equals, bit for bit,
that of the same film stepped with no tile left out as still, at a fixed dt on
both sides of the substep limit and with dt chosen on the device."""
import numpy as np
import pytest

import pyoracle as po
from canvaz_film import capi, synth
from test_gpu_still import PLANES, strokes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(208, 160), (207, 150)])
@pytest.mark.parametrize("awake", [1, 0])
@pytest.mark.parametrize("substeps", [1, 9, 0])  # 0: cf_step_adaptive
def test_still_tiles_change_nothing_around_implicit_steps(w, h, awake, substeps):
    import __graft_entry__ as g
    g.build()
    from canvaz_film.film import Film
    cv = synth.blob_canvas(w, h, 11, n_blobs=2, sigma=(3, 6), per_cell_n=False, tables="reference", tau=(0.0, 0.3),
                           mu=(0.05, 0.2), peak_mm=(3.0, 5.0))
    cv.settings.update(implicit_hydro=1, all_active=awake)
    st = po.make_settings(cv.settings)
    dx = float(st.width_m) / w
    films = [Film(st, w, h, capi.CF_PREC_FP32) for _ in range(2)]
    for f in films:
        f.set_tables(cv.pigtab, cv.cmf)
        f.write_state(cv.planes)
        f.update_params(1 / 60, max(substeps, 1))
    before = films[0].read_state()["h"]
    for k in range(12):
        for f, forget in zip(films, (False, True)):
            if substeps:
                f.update_params(1 / 60, substeps)
            if k in (4, 8):
                f.upload_deposits(np.array(strokes(dx, [(150, 120), (20 + 10 * k, 20)])))
            if forget:
                f.set_params(f.params())
            if substeps:
                f.encode_frame(substeps)
            else:
                f.step_adaptive(1 / 60)
            f.sync()
        for p in PLANES:
            a, b = films[0].plane(p), films[1].plane(p)
            assert np.array_equal(a, b, equal_nan=True), (k, p, np.flatnonzero(a != b)[:8])
    assert not np.array_equal(films[0].read_state()["h"], before)
    films[0].stats()  # raises where a wait ran out
