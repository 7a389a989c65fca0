"""The launch autotuner beside the split launches of heavily contracted quartets: candidates compared on the
whole work of a class, and nothing recorded where there is nothing to choose."""
import re

import numpy as np
import pytest
import torch

from lible_b200 import ints as L
from lible_b200.workloads import random_density, water_cluster

pytestmark = pytest.mark.gpu


def _times(summary):
    return {m[0]: float(m[1]) for m in re.findall(r"^\((\d\d\|\d\d)\) fp64 .* ([\d.e+]+) ms$", summary, re.M)}


def test_candidates_are_timed_with_their_split_launch():
    """(ss|ss) of one water: nearly all of its time is the split launch of the two core pairs, 64 x 64
    primitive pairs a quartet.  The time of the chosen candidate covers it: at least half of what a
    profiled build spends on the class."""
    Z, xyz, rng = water_cluster(1, seed=51)
    s = L.Structure("cc-pvdz", Z, xyz, units="bohr")
    D = random_density(s.nao, 5, rng)
    J, K, _ = L.jk(s, D)
    times = _times(L.jk_autotune(s, D))
    runs = [L.jk_profile(s, D) for _ in range(5)]
    ms = min(r["ms"] for p in runs for r in p if r["classes"] == (0, 0, 0, 0))
    assert times["00|00"] >= 0.5 * ms
    Jt, Kt, _ = L.jk(s, D)
    assert np.abs(Jt - J).max() <= 1e-12 and np.abs(Kt - K).max() <= 1e-12


def test_a_class_without_an_ordinary_launch_leaves_no_entry(tmp_path):
    """Two atoms with one contraction of six s functions each: every quartet goes to the split launch."""
    shell = (0, [40.0, 12.0, 4.0, 1.5, 0.6, 0.25], [0.02, 0.1, 0.3, 0.4, 0.3, 0.1])
    s = L.Structure([[shell], [shell]], [2, 2], [[0.0, 0.0, 0.0], [0.0, 0.0, 1.4]], units="bohr")
    D = np.array([[1.0, 0.3], [0.3, 0.8]])
    J, K, st = L.jk(s, D, schwarz=0.0)
    assert st["n_quartets"] == 6
    cache = tmp_path / "tune.txt"
    assert _times(L.jk_autotune(s, D, schwarz=0.0, cache=str(cache))) == {}
    assert cache.read_text() == ""
    Jt, Kt, _ = L.jk(s, D, schwarz=0.0)
    assert np.abs(Jt - J).max() <= 1e-12 and np.abs(Kt - K).max() <= 1e-12


def test_choices_of_older_kernels_are_not_taken_over(tmp_path):
    """A cache whose lines name the GPU alone, as before the warp and split forms, with the other orientation
    for every class."""
    Z, xyz, rng = water_cluster(1, seed=52)
    s = L.Structure("cc-pvtz", Z, xyz, units="bohr")
    D = random_density(s.nao, 5, rng)
    cache = tmp_path / "tune.txt"
    L.jk_autotune(s, D, cache=str(cache))
    gpu = torch.cuda.get_device_name(0)
    lines = cache.read_text().splitlines()
    assert lines and all(x.startswith(gpu) for x in lines)
    old = [f"{gpu}|{x.split('|', 1)[1].rsplit(' ', 1)[0]} 2" for x in lines]
    cache.write_text("\n".join(old) + "\n")
    s2 = L.Structure("cc-pvtz", Z, xyz, units="bohr")
    L.set_tune_cache(s2, str(cache))
    assert {r["shape"] for r in L.jk_profile(s2, D)} == {0}
