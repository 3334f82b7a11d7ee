"""The knobs a batch is tuned for are those its launches read (CPU: no launch)."""
import types

import pytest

from euvlitho_b200 import _lib as L
from euvlitho_b200 import autotune as A
from euvlitho_b200 import build


@pytest.mark.parametrize("precision,orders,sources,pixels,lp,split,rows", [
    (L.EUV_PREC_MIXED, 121, 8, 64, 4, True, True),      # FP64 products below 128 orders
    (L.EUV_PREC_MIXED, 129, 8, 64, 4, True, False),
    (L.EUV_PREC_FP64, 961, 200, 256, 20, False, True),  # band-limited image
    (L.EUV_PREC_MIXED, 961, 200, 256, 20, False, False),
])
def test_shapes_hold_the_knobs_in_use(precision, orders, sources, pixels, lp, split, rows):
    build.build()
    d = L.AbbeDesc()
    d.xdiv = d.ydiv = pixels
    d.lpx = d.lpy = lp
    d.n_units, d.n_src, d.precision = 24, sources, precision
    batch = types.SimpleNamespace(
        plan=types.SimpleNamespace(precision=precision, orders=types.SimpleNamespace(n=orders)),
        U=24, ax=types.SimpleNamespace(shape=(24, sources, orders)), adesc=d)
    sh = A.shapes(batch)
    assert ("abbe_split" in sh) == split
    assert ("zgemm_rows" in sh) == rows
    assert sh["lu_cluster"] == [(orders, 24)]


def test_header_and_binding_agree_on_the_fp64_orders():
    import os
    import re
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    txt = open(os.path.join(root, "include", "euvl_b200.h")).read()
    assert int(re.search(r"EUV_MIXED_FP64_ORDERS (\d+)", txt).group(1)) == L.EUV_MIXED_FP64_ORDERS
