"""The dense FP64 kernel's work split, on the host: every tile is dealt once, and
the splits that measurements on 148 SMs have shown to be the faster ones."""
import random

import pytest

import tblis_b200 as tb


def tiles(p, m, n, l, cplx):
    if p["exchanged"]:
        m, n = n, m
    bm, bn = p["tile"]
    return -(-m // bm) * -(-(2 * n if cplx else n) // bn) * l


@pytest.mark.parametrize("seed", range(200))
def test_every_tile_once(seed):
    r = random.Random(seed)
    m, n, k = (int(2 ** r.uniform(0, 14)) for _ in range(3))
    l = r.choice([1, 1, 1, int(2 ** r.uniform(0, 12))])
    cplx, beta = r.random() < 0.4, r.choice([0.0, 1.0])
    p = tb.dense_plan(m, n, k, l, cplx, beta)
    assert p["whole"] + p["cut_tiles"] == tiles(p, m, n, l, cplx)
    assert p["cut"] == (p["cut_tiles"] > 0) and 1 <= p["ctas"] <= 148
    # whole waves stay whole: every CTA has as many
    assert p["whole"] % 148 == 0 or not p["cut"]


# 148 SMs, FP64, us uncut and cut (128 x 128 tiles): 2000 x 2000 x 200 77 and 98, 3000 x
# 1500 x 300 105 and 130, 100 matrices of 300^3 238 and 379, 1000 of 100 x 100 x 300
# 312 and 528; 40000 x 100 x 500 217 and 190, 97 x 97 x 93217 one tile
@pytest.mark.parametrize("m,n,k,l,cut", [
    (2000, 2000, 200, 1, False), (3000, 1500, 300, 1, False), (4000, 4000, 64, 1, False), (300, 300, 300, 100, False),
    (100, 100, 300, 1000, False), (20, 200, 1000, 100, False), (1000, 60, 1000, 100, False),
    (40000, 100, 500, 1, True), (97, 97, 93217, 1, True), (300, 300, 30000, 2, True)])
def test_cut(m, n, k, l, cut):
    assert tb.dense_plan(m, n, k, l)["cut"] == cut
