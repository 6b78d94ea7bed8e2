"""The implicit step's solve (one cooperative launch) at the sizes where its
walk over the tiles can go wrong: fewer tiles than one block takes, counts that
leave a span or a group short, ragged edges, tiles without paint or asleep;
and batches large enough for the per-film sums to be spread over the blocks."""
import numpy as np
import pytest

import parity
import pyoracle as po
from canvaz_film import capi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built():
    import __graft_entry__ as g
    g.build()
    return True


def pour(w, h, seed, blobs):
    cv = synth.blob_canvas(w, h, seed, n_blobs=blobs, sigma=(3, 6), per_cell_n=False, tables="reference",
                           tau=(0.0, 0.3), mu=(0.05, 0.2), peak_mm=(3.0, 5.0))
    cv.settings.update(implicit_hydro=1)
    return cv


# 1 tile; 6 ragged tiles; 39 tiles of one column pair; 5 of one row; paint in a corner of 1024 tiles
@pytest.mark.parametrize("w,h,blobs", [(16, 16, 1), (33, 17, 2), (40, 200, 5), (70, 16, 2), (512, 512, 2)])
def test_solve_vs_oracle(built, w, h, blobs):
    """h within 1e-5 of FP64, or 1.5x the FP32 mirror's own distance."""
    from canvaz_film.film import Film
    cv = pour(w, h, w + h, blobs)
    st = po.make_settings(cv.settings)
    runs = [po.Oracle(w, h, st, 1, 64), po.Oracle(w, h, st, 1, 32), Film(st, w, h, capi.CF_PREC_FP32)]
    for x in runs:
        x.set_tables(cv.pigtab, cv.cmf)
        x.write_state(cv.planes)
    steps = []
    for _ in range(3):
        n = runs[0].choose_substeps(1 / 60)
        for x in runs:
            x.update_params(1 / 60, n)
        steps.append(runs[0].implicit_steps())
        for x in runs:
            x.encode_frame(n)
        runs[2].sync()  # the next update_params takes its step count from this frame's stats
    assert max(steps) > 0, steps  # the solve ran
    assert runs[2].stats()["wet_cells"] > 0  # stats also report a wait that ran out
    h64, h32, hg = runs[0].buf("h"), runs[1].buf("h"), runs[2].read_state()["h"]
    assert parity.rel_l2(hg, h64) <= max(parity.H_REL_L2, 1.5 * parity.rel_l2(h32, h64))


@pytest.mark.parametrize("films", [2, 5, 9])
def test_solve_of_many_films_equals_alone(built, films):
    """A batch's solve sums each film's partials as the film alone does, bit
    for bit, whatever shares the launch."""
    from canvaz_film.film import Batch, Film
    alone, batched = [], []
    for k in range(films):
        cv = pour(20 + 13 * k, 61 - 5 * k, k, 2)
        for lst in (alone, batched):
            f = Film(po.make_settings(cv.settings), cv.w, cv.h, capi.CF_PREC_FP32)
            f.set_tables(cv.pigtab, cv.cmf)
            f.write_state(cv.planes)
            f.update_params(1 / 60, 4)
            lst.append(f)
    b = Batch()
    for f in batched:
        b.add(f)
    b.step(2, 4)
    for f in alone:
        f.encode_frame(4)
        f.encode_frame(4)
    for fa, fb in zip(alone, batched):
        fa.sync()
        fb.sync()
        ha, hb = fa.read_state()["h"], fb.read_state()["h"]
        assert np.array_equal(ha.view(np.uint32), hb.view(np.uint32))


@pytest.mark.parametrize("order", [(0, 1), (0, 0, 1, 0, 1), (1, 0)])
def test_films_without_implicit_steps_share_a_batch(built, order):
    """Films with implicit_hydro off (they hold no CG planes), before, among
    and after films whose frames take implicit steps: each as alone, bit for
    bit."""
    from canvaz_film.film import Batch, Film
    alone, batched = [], []
    for k, implicit in enumerate(order):
        cv = pour(40 + 9 * k, 50, k, 2)
        cv.settings.update(implicit_hydro=implicit)
        for lst in (alone, batched):
            f = Film(po.make_settings(cv.settings), cv.w, cv.h, capi.CF_PREC_FP32)
            f.set_tables(cv.pigtab, cv.cmf)
            f.write_state(cv.planes)
            f.update_params(1 / 60, 4)
            lst.append(f)
    b = Batch()
    for f in batched:
        b.add(f)
    b.step(2, 4)
    for f in alone:
        f.encode_frame(4)
        f.encode_frame(4)
    for fa, fb in zip(alone, batched):
        assert fb.stats()["wet_cells"] > 0
        fa.sync()
        ha, hb = fa.read_state()["h"], fb.read_state()["h"]
        assert np.array_equal(ha.view(np.uint32), hb.view(np.uint32))
    b.close()


@pytest.mark.parametrize("films", [1, 3])
def test_a_solve_that_gives_up_is_reported_by_every_film(built, films):
    """With a limit of no polls the first block to wait at a meeting leaves the
    solve and the others follow: the kernel returns, every film of the launch
    reports the timeout and keeps its h through the implicit step, and the next
    frame, with the default limit, solves as a film that never gave up."""
    from canvaz_film.film import Batch, Film
    fs, ref, keep = [], [], []
    for k in range(films):
        cv = pour(150 + 16 * k, 130, k, 4)  # 90 tiles and more: 12 or more blocks
        cv.settings.update(all_active=1)
        for lst in (fs, ref, keep):
            st = po.make_settings(dict(cv.settings, implicit_hydro=int(lst is not keep)))
            f = Film(st, cv.w, cv.h, capi.CF_PREC_FP32)
            f.set_tables(cv.pigtab, cv.cmf)
            f.write_state(cv.planes)
            f.update_params(1 / 60, 1)
            lst.append(f)

    def step(lst):
        b = Batch()  # a batch captures its frames with the limit of the time
        for f in lst:
            b.add(f)
        b.step(1, 1)
        for f in lst:
            f.sync()
        b.close()

    for f in fs:
        f.set_wait_limit(0)
    step(fs)
    for f in fs:
        with pytest.raises(capi.FilmError) as e:
            f.stats()
        assert e.value.status == capi.CF_ERR_TIMEOUT
    step(keep)  # the same frame of films that take no implicit steps
    step(ref)
    for f, g, r in zip(fs, keep, ref):
        h = f.read_state()["h"]
        assert np.array_equal(h, g.read_state()["h"])
        assert not np.array_equal(h, r.read_state()["h"])
    # later frames: those of a film that is written the same state
    for f, g in zip(fs, ref):
        g.write_state(f.read_state())
        s = f.read_state()
        f.write_state(s)
        for x in (f, g):
            x.set_wait_limit(1 << 22)
            x.update_params(1 / 60, 1)
    step(fs)
    step(ref)
    for f, g in zip(fs, ref):
        assert g.stats()["wet_cells"] > 0
        assert np.array_equal(f.read_state()["h"], g.read_state()["h"])
