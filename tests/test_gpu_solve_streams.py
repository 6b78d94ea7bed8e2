"""The implicit solve, one cooperative launch, where it does not have the chip
to itself: films stepped at the same time on streams of their own, and a film
stepped on a stream that has a part of the SMs (a green context)."""
import ctypes as C

import numpy as np
import pytest

import pyoracle as po
from canvaz_film import capi, synth

pytestmark = pytest.mark.gpu


def pour_film(seed, w=720, h=560):
    """1575 tiles: more than the solve's blocks hold at a time."""
    import __graft_entry__ as g
    g.build()
    from canvaz_film.film import Film
    cv = synth.blob_canvas(w, h, seed, n_blobs=24, sigma=(5, 25), per_cell_n=False, tables="reference",
                           tau=(0.0, 0.3), mu=(0.05, 0.2), peak_mm=(3.0, 5.0))
    cv.settings.update(implicit_hydro=1)
    f = Film(po.make_settings(cv.settings), cv.w, cv.h, capi.CF_PREC_FP32)
    f.set_tables(cv.pigtab, cv.cmf)
    f.write_state(cv.planes)
    f.update_params(1 / 60, 4)
    return f


def bits(f):
    f.stats()  # raises where a wait ran out
    return f.read_state()["h"].view(np.uint32)


def test_films_on_streams_of_their_own():
    import torch
    want, fs = [], [pour_film(s) for s in (1, 2, 3)]
    for s in (1, 2, 3):
        f = pour_film(s)
        for _ in range(3):
            f.encode_frame(4)
        want.append(bits(f))
    streams = [torch.cuda.Stream() for _ in fs]
    torch.cuda.synchronize()
    for _ in range(3):
        for f, st in zip(fs, streams):
            f.encode_frame(4, st.cuda_stream)
    torch.cuda.synchronize()
    for f, w in zip(fs, want):
        assert np.array_equal(bits(f), w)


def green_stream(min_sms):
    """A stream on at least min_sms SMs and how many it has (CUDA driver API)."""
    cu = C.CDLL("libcuda.so.1")
    res, part, rest = (C.create_string_buffer(256) for _ in range(3))  # CUdevResource
    n, desc, ctx, st, dev = C.c_uint(1), C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_int()
    for name, *args in (("cuDeviceGet", C.byref(dev), C.c_int(0)),
                        ("cuDeviceGetDevResource", dev, res, C.c_int(1)),
                        ("cuDevSmResourceSplitByCount", part, C.byref(n), res, rest, C.c_uint(0), C.c_uint(min_sms)),
                        ("cuDevResourceGenerateDesc", C.byref(desc), part, C.c_uint(1)),
                        ("cuGreenCtxCreate", C.byref(ctx), desc, dev, C.c_uint(1)),
                        ("cuGreenCtxStreamCreate", C.byref(st), ctx, C.c_uint(1), C.c_int(0))):
        if not hasattr(cu, name):
            pytest.skip("the driver has no " + name)
        status = getattr(cu, name)(*args)
        assert status == 0, (name, status)
    return st.value, C.c_uint.from_buffer(part, 96).value


def test_a_film_on_a_part_of_the_sms():
    import torch
    whole, part = pour_film(5), pour_film(5)
    st, sms = green_stream(16)
    assert 16 <= sms < torch.cuda.get_device_properties(0).multi_processor_count
    torch.cuda.synchronize()
    for f, stream in ((whole, None), (part, st)):
        for _ in range(3):
            f.encode_frame(4, stream)
        torch.cuda.synchronize()
    assert np.array_equal(bits(part), bits(whole))
