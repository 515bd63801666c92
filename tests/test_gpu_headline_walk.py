"""The default form (the walk) against the oracle at the shape the benchmark times, by
the checks of the other two forms."""
from __future__ import annotations

import pytest

import test_gpu_headline as headline
from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu


def test_default_form_graph_training_equals_oracle_every_iteration(hand_table):
    headline.test_graph_training_equals_oracle_every_iteration(hand_table, L.FORM_AUTO)


def test_default_form_full_size_update_equals_oracle(hand_table):
    headline.test_full_size_update_equals_oracle(hand_table, L.FORM_AUTO)
