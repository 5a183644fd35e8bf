"""The autotuner leaves out what no kernel reads: tile widths and radix orders of
axes whose transforms have a fixed shape, and widths beyond the grid's lines."""
import json

import pytest

from deft_gb300 import _lib, autotune

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision,fixed", [
    (36, 1, [True, True, False]), (24, 1, [False] * 3), (256, 1, [True, True, False]),
    (64, 0, [True, True, False]), (32, 0, [False] * 3), (48, 0, [False] * 3)])
def test_fixed_axes(n, precision, fixed):
    shape = (n, n, n) if n < 256 else (256, 256, 32)
    b = autotune._Bench(shape, precision)
    try:
        tiles, radix = b.tiles()
        assert [b.fixed(a, shape[a]) for a in range(3)] == fixed
        t2, r2 = b.tiles()
        assert list(t2) == list(tiles) and list(r2) == list(radix)
    finally:
        b.close()


def test_entry_of_fixed_axes():
    e = autotune.tune((36, 36, 36), _lib.PRECISION_MIXED, repeats=1, trials=1)
    assert e["tiles"][0] == e["tiles"][2] == e["tiles"][3] == 0 and not any(e["radix"][:16])
    assert e["tiles"][4] > 0 and e["tiles"][5] > 0 and any(e["radix"][16:])


def test_entry_is_what_takes_effect(monkeypatch):
    # 24 x 13 lines along y: 13 columns are all there are
    monkeypatch.setattr(autotune, "CANDIDATES", (13, 24, 64))
    e = autotune.tune((24, 24, 24), _lib.PRECISION_MIXED, repeats=1, trials=1)
    assert e["tiles"][0] == 13


def test_bundled_entries():
    with open(autotune.BUNDLED) as f:
        entries = json.load(f)["entries"]
    for e in entries:
        b = autotune._Bench(tuple(e["N"]), e["precision"])
        try:
            for a in (0, 1):
                if b.fixed(a, e["N"][a]):
                    assert not any(e["radix"][8 * a:8 * a + 8]), e["N"]
                    for p in autotune.AXIS_PARAMS[a]:
                        assert e["tiles"][autotune.PARAMS.index(p)] == 0, e["N"]
        finally:
            b.close()
