"""What the TF32x3 GEMM launcher makes of its plan, through ct_tc_gemm_form (no GPU): 64-wide tiles where
128-wide ones would leave half of the SMs idle, pairs of CTAs on whole wide tiles.  The launcher
decides by the same two functions.
"""
import ctypes as C

import numpy as np
import pytest

from test_host_tc_plan import defaults, lib, plan  # noqa: F401  (fixtures: the built library, no switches set)


def form(lib, m, n, k, sms=152):  # noqa: F811
    out = (C.c_int64 * 3)()
    assert lib.ct_tc_gemm_form(m, n, k, sms, out) == 0
    return tuple(out)


def test_narrow_tiles_at_their_edge(lib, monkeypatch):  # noqa: F811
    # 19 rows of tiles: 8 halves per row fill 152 SMs, 9 do not
    assert form(lib, 19 * 128, 512, 160) == (64, 1, 152)
    assert form(lib, 19 * 128, 513, 160)[0] != 64
    assert form(lib, 1, 1, 1) == (64, 1, 1)
    monkeypatch.setenv("CTDMRG_TC_BN", "128")
    assert form(lib, 19 * 128, 512, 160)[0] == 128
    monkeypatch.delenv("CTDMRG_TC_BN")
    monkeypatch.setenv("CTDMRG_TC_KCHUNK", "0")
    assert form(lib, 19 * 128, 512, 160)[:2] in ((128, 1), (256, 1))


def test_pairs_at_their_edges(lib, monkeypatch):  # noqa: F811
    assert form(lib, 5120, 4096, 1024) == (224, 2, 152)      # H_eff's first product at chi 1024
    assert form(lib, 4096, 1024, 5120) == (224, 2, 152)      # its last one, transposed: 8 rows of tiles
    assert form(lib, 5120, 4096, 992)[1] == 1                # less deep
    assert form(lib, 5120, 4096, 993)[1] == 2                # 993 is padded to 1024
    assert form(lib, 4096, 1024, 5120, 151)[1] == 1          # an odd number of SMs
    assert plan(lib, 8192, 2048, 8192)["gsk"] > 0 and form(lib, 8192, 2048, 8192)[1] == 1   # a stream-K last wave
    monkeypatch.setenv("CTDMRG_TC_KCHUNK", "0")
    assert form(lib, 5120, 4096, 1024)[1] == 1


@pytest.mark.parametrize("sms", [152, 148, 131])
def test_form_follows_the_plan(lib, sms):  # noqa: F811
    rng = np.random.default_rng(sms)
    seen = set()
    for _ in range(400):
        m, n, k = (int(np.exp(rng.uniform(0, np.log(9000)))) for _ in range(3))
        p, (bn, ctas, grid) = plan(lib, m, n, k, sms), form(lib, m, n, k, sms)
        rows, cols = (n, m) if p["trans"] else (m, n)
        tiles = -(-rows // 128) * -(-cols // bn)
        halves = -(-rows // 128) * -(-cols // 64) <= sms
        assert bn == (64 if p["bn"] == 128 and halves else p["bn"])
        pair = bn >= 224 and p["gsk"] == 0 and -(-rows // 128) % 2 == 0 and p["nkb"] >= 32 and sms % 2 == 0
        assert ctas == (2 if pair else 1)
        assert grid == (2 * min(tiles // 2, sms // 2) if pair else min(tiles, sms))
        seen.add((bn, ctas))
    assert (64, 1) in seen and (sms != 152 or seen & {(224, 2), (256, 2)})
