"""The autotuners time only what the batch's forces read: threads per block and per
particle of the mixed traversal above XNB_MIXED_SPLIT_MAX particles. Elsewhere the
trials would run the same kernels and noise would pick the winner."""
import pytest

from exanbody_gb300 import ensemble, workloads, xnb
from helpers import ncells, new_batch

FORCE = ("force_block", "force_lanes")


@pytest.mark.parametrize("atoms,precision,searched", [
    ([30000, 20000], xnb.PREC_MIXED, False),
    ([30000, 20001], xnb.PREC_MIXED, True),
    ([30000, 2000000], xnb.PREC_FP64, False),
])
def test_ensemble_trials(monkeypatch, atoms, precision, searched):
    calls = []

    def trial(systems, cfg, steps, precision, stream):
        calls.append(dict(cfg))
        return float(len(calls))  # the last one tried always leads

    monkeypatch.setattr(ensemble, "trial", trial)
    best, _, log = ensemble.autotune([{"n_atoms": n} for n in atoms], precision, steps=5, stream=object())
    for key in FORCE:
        assert len({c[key] for c in calls}) == (3 if searched else 1)
        assert searched or best[key] == ensemble.DEFAULTS[key]
    assert len(log) == len(calls) == (9 if searched else 5)


@pytest.mark.gpu
@pytest.mark.parametrize("n,precision,trials", [
    (10, xnb.PREC_MIXED, 5),   # the present setting, the other build form, two stages, the half lists
    (10, xnb.PREC_FP64, 5),
    (24, xnb.PREC_MIXED, 9),   # and two block sizes, two numbers of threads per particle
    (24, xnb.PREC_FP64, 5),
])
def test_native_trials(n, precision, trials):
    w = workloads.lj_fcc_system(n, 0.8442, 1.0, 3)
    b = new_batch([w["n_atoms"]], [ncells(w["geom"])])
    s = b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"])
    b.set_tuning(640, 128)
    b.set_force_lanes(2)
    b.init_particles(s, precision)
    t = b.autotune(3, precision)
    assert t["trials"] == trials
    if trials == 5:
        assert (t["force_block"], t["force_lanes"]) == (128, 2)
    b.close()
