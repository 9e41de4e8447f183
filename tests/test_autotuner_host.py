"""The autotuners' default candidates: options without an effect are not tried twice (no GPU)."""
import itertools

from distorteddustydiscanalysistoolkits_b200 import batch


def test_inert_options_are_tried_once():
    for tuner, settings in ((batch.Autotuner(), 6), (batch.BatchAutotuner(), 16)):
        assert len(tuner.grid["walk_split"]) == 1
        assert len(list(itertools.product(*tuner.grid.values()))) == settings
