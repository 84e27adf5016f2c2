"""Kernels at the edges of their tiles and of the rules that choose them, against the plain statements and the oracle."""
import numpy as np
import pytest

import lm_plain as plain
from lm_models import LIMIT, Case, attention, config, delta, error, feed, tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 32, 33, 64, 65])
def test_float32_gemm_rows(pkg, tmp_path, rows):
    """Portions on both sides of the few-rows kernel's and the tile kernel's edges; widths that split K (above 1024)
    and that end inside a step of 32 columns. The limit is the 32-bit mode's: summation order."""
    c = Case(pkg, tmp_path, config([delta(ff=1300), attention(ff=60)], width=1100, vocab=301), seed=rows)
    toks = tokens(c.cfg, rows + 70, rows)
    want = plain.forward(c.w, c.cfg, toks)[0]
    with c.open("float32") as lm:
        s = lm.open()
        assert error(feed(lm, s, toks, [rows, 70]), want) < LIMIT["float32"]
