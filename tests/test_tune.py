"""The launch knobs as Python sees them, and what the batch tuner tries."""
import pytest


@pytest.mark.parametrize("value", [0.0, 0.4, 0.75, 1.5, 3.0, 0.1, 63.99])
def test_light_factor_reads_back_as_it_was_set(ecl, value):
    """The knob is a C float: 0.4 comes back as 0.4, here and through the library."""
    t = ecl.Tune()
    t.mst_light_factor = value
    assert t.mst_light_factor == value and t.as_dict()["mst_light_factor"] == value
    old = ecl.set_tune(mst_light_factor=value)
    try:
        assert ecl.get_tune().mst_light_factor == value
    finally:
        ecl.set_tune(old)
    assert ecl.Tune(8).blocks_per_sm == 8 and len(t.as_dict()) == 10


@pytest.mark.gpu
@pytest.mark.parametrize("degree", [6, 40])  # on both sides of the default's rule
def test_tuner_tries_every_candidate(ecl, orc, degree):
    """One point for the start, one for each other value of each knob that the
    batch's codes have: 4 grid sizes, 4 light factors, 3 + 4 row thresholds."""
    b = ecl.Batch()
    for k in range(4):
        b.add(ecl.gen_er(2000, degree / 2000, seed=k, symmetrise=True, weight_seed=k + 1))
    b.build(ecl.BATCH_CC | ecl.BATCH_MST)
    t = b.tune(trials=1)
    assert b.tune_points == 1 + 3 + 3 + 2 + 3
    assert t.mst_light_factor in (0.75, 1.5, 3.0, 0.4)
    b.run()
    assert b.result(0, ecl.BATCH_MST)[1] == orc.mst(b.graph(0))[1]
