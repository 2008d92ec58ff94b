"""Operators of the mixed form driven from several host threads of the caller's
own. Their correction loops are CUDA graphs only where a thread is alone in
the library (csrc/call_gate.cuh, tests/cpp/call_gate.cu), so the threads'
runs must end, and give what the runs one by one give."""

import os
import subprocess
import threading

import numpy as np
import pytest

from tests import _native


def test_the_gate_without_a_device():
    result = subprocess.run([str(_native.build("call_gate.cu"))], capture_output=True, text=True, timeout=300,
                            env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    print(result.stdout)
    assert result.returncode == 0, result.stdout + result.stderr


@pytest.mark.gpu
def test_gpu_mixed_operators_in_the_callers_threads(gpu):
    from sl3dpp_gb300.ensemble import Ensemble, ensemble_members

    members = ensemble_members(4, seed=11, steps=3, lmax_choices=(8, 12))
    for m in members:
        m["elements"] = 20
    want = Ensemble(members, precision=1).run_sequential()
    rounds = 3
    own = [[Ensemble([m], precision=1) for m in members] for _ in range(rounds)]
    got = [[None] * len(members) for _ in range(rounds)]
    failed = []

    def drive(k):
        try:
            for r in range(rounds):  # run and destroyed beside the others' calls
                got[r][k] = own[r][k].run_sequential()
                got[r][k].pop("states")
                own[r][k] = None
        except BaseException as e:  # noqa: BLE001 -- reported below
            failed.append(e)

    threads = [threading.Thread(target=drive, args=(k,)) for k in range(len(members))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for k in range(len(members)):
        for key in ("U", "phi"):
            for r in range(rounds):
                a, b = got[r][k][key][0], want[key][k]
                assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b)), (r, k, key)
