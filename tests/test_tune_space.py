"""CPU: the autotuner searches only parameters that change a launch."""
from adeco_gb300 import tune


def test_parameters_without_effect_are_not_searched():
    assert all("share_chunk" not in space for space in tune.SPACES.values())
    assert tune.DEFAULTS["share_chunk"] == 512  # still accepted, and in saved settings
    measured = []
    best, _, _ = tune.search(tune.SPACES["zoom"], lambda p: measured.append(p) or 1.0)
    assert best == {k: tune.DEFAULTS[k] for k in tune.SPACES["zoom"]}
    assert len(measured) == 1 + sum(len(v) - 1 for v in tune.SPACES["zoom"].values())
