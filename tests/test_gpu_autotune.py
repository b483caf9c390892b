"""The tile tuner measures the launches that a step makes: the fluxes of both
directions of all instances in one launch, and the cell update of all instances. And
shapes that a cache file holds from other kernels are measured again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(rh, sizes):
    fields = [rh.cases.init_cylinder(h=3.0 / (nx - 1)) for nx in sizes]
    return rh.Batch(fields, [rh.GhostGrid.build(f) for f in fields], exact=True)


def test_times_are_the_steps(rh):
    """sizes of no other test (the process keeps the shapes of a class)"""
    b = _batch(rh, (87, 87, 127, 127, 127, 127))
    lg = [b.tile_shapes(k) for k in (0, 2)]
    steps = [b.profile_steps(2, 0.05) for _ in range(5)]
    flux, rhs = (min(p[n][0] for p in steps) / 6 for n in ("flux", "rhs_stage"))
    res = b.autotune(reps=5)
    assert len(res) == 2
    for e, s in zip(res, lg):
        for ms, k in ((e["ms_fx"], s[0] - 2), (e["ms_fy"], s[1] - 4)):
            assert 0.75 * flux <= ms[k] <= 1.25 * flux, (ms, flux)
        # (the timed cell update writes the rhs alone, not the stage's state)
        assert 0.6 * rhs <= e["ms_rhs"][s[2] - 4] <= 1.25 * rhs, (e["ms_rhs"], rhs)
    assert res[0]["ms_fx"][lg[0][0] - 2] == res[0]["ms_fy"][lg[0][1] - 4] or res[0]["shape"][0] != lg[0][0]
    # a shape that is applied beat the default by 3%
    for e, s in zip(res, lg):
        for ms, k, d in ((e["ms_fx"], e["shape"][0] - 2, s[0] - 2), (e["ms_fy"], e["shape"][1] - 4, s[1] - 4),
                         (e["ms_rhs"], e["shape"][2] - 4, s[2] - 4)):
            assert k == d or ms[k] < 0.97 * ms[d]
    assert [b.tile_shapes(k) for k in (0, 2)] == [e["shape"] for e in res]
    b.close()


def test_cache_of_other_kernels_is_measured_again(rh, tmp_path):
    path = tmp_path / "tiles.txt"
    path.write_text("71 281 0 4 6 6\n")
    b = _batch(rh, (71,))
    assert b.tile_shapes(0) != (4, 6, 6)
    res = b.autotune(cache_path=str(path), reps=2)
    assert not res[0]["from_cache"] and min(res[0]["ms_fx"]) > 0
    text = path.read_text().split("\n")
    assert text[0] == "rh3t tile shapes 2" and "71 281 0 %d %d %d" % res[0]["shape"] in text
    assert b.autotune(cache_path=str(path))[0]["from_cache"]
    b.close()


def test_tuned_and_untuned_agree(rh):
    a, b = _batch(rh, (41, 53, 67)), _batch(rh, (41, 53, 67))
    b.autotune(reps=2)
    for q in (a, b):
        q.advance(5, 0.05)
    assert np.array_equal(a.download_values()[0], b.download_values()[0])
    a.close()
    b.close()
