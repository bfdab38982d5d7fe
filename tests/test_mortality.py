"""The step's mortality, on the host: the larvae's hourly mortality in
binary32 against its binary64 definition (every 7th input here; the same
program with stride 1 enumerates the whole domains), and the kill threshold
and whole-hour days of sampo_model.cuh against the comparisons they stand for."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sampo_gb300", "csrc")
F = np.float32


def _run(tmp_path, source, name, *args, cxx="gcc"):
    cc = shutil.which(cxx)
    if cc is None:
        pytest.skip(f"{cxx} not available")
    exe = str(tmp_path / name)
    subprocess.run([cc, "-O2", "-ffp-contract=off", "-fopenmp", "-I", CSRC, source, "-o", exe, "-lm"], check=True)
    out = subprocess.run([exe, *args], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout


def test_larval_mortality_equals_its_definition(tmp_path):
    out = _run(tmp_path, os.path.join(HERE, "mortality_check.c"), "mortality_check", "7")
    lines = {l.split()[0]: l for l in out.splitlines() if l.strip()}
    # the pairs' measured errors stay below their bounds with the margin the bounds assume
    for fn, bound in (("exp", -40), ("pow", -38)):
        assert "mismatches=0" in lines[fn], lines[fn]
        assert float(re.search(r"maxrel=2\^(-?[\d.]+)", lines[fn]).group(1)) <= bound - 2, lines[fn]
    assert lines["hmr"].endswith("mismatches=0")


def kill_threshold(hmr):
    """kill_threshold (sampo_model.cuh), vectorised."""
    h = (hmr * F(4294967296.0)).astype(np.float64)
    n = h.astype(np.uint64)
    half = np.maximum(np.exp2(np.floor(np.log2(np.maximum(h, 1.0))) - 24), 1).astype(np.uint64)
    big = n + half + np.where((n // (2 * half)) % 2 == 1, 0, 1).astype(np.uint64)
    return np.where(h < 16777216.0, n + 1, big)


def test_kill_threshold_is_the_comparison():
    """(float)v * 2^-32 <= hmr exactly for v < kill_threshold(hmr)."""
    rng = np.random.default_rng(1)
    hmr = np.concatenate([rng.uniform(0, 0.98, 20000), 2.0 ** -np.arange(1, 33), rng.uniform(0, 2.0 ** -8, 20000), [0.0]]).astype(F)
    t = kill_threshold(hmr).astype(np.int64)
    for d in (-600, -129, -2, -1, 0, 1, 2, 128, 600):
        v = t + d
        ok = (v >= 0) & (v <= 0xFFFFFFFF)
        dies = F(2.3283064365387e-10) * v[ok].astype(np.uint32).astype(F) <= hmr[ok]
        assert np.array_equal(dies, d < 0 * v[ok]), d


def test_whole_hours_give_the_same_days():
    """whole_age_days (sampo_model.cuh) for every whole age below 2^21 hours."""
    age = np.arange(1 << 21, dtype=F)
    q = (age + F(0.5)) * F(1.0 / 24.0)
    assert np.array_equal(q.astype(np.uint32), (age / F(24.0)).astype(np.uint32))
    # and an hour on, from the same quotient
    assert np.array_equal((q + F(1.0 / 24.0)).astype(np.uint32)[:-1], (age[1:] / F(24.0)).astype(np.uint32))
