"""The kernels that the benchmark says a step launches, against the sequence of
launch_step (csrc/stage.cu) written out, and 13 for a refined mesh with ghosts,
as a profiler's launch list of such a step has it."""
import pytest

import bench


def _sequence(wls, restrict, ghosts):
    seq = ["begin"] if wls + restrict else ["control"]
    for stage in (1, 2, 3):
        if wls + restrict:
            seq += ([] if stage == 1 else ["requests"]) + (["restrict"] if restrict else [])
        seq += ["faces", "cells"] + (["ghosts"] if ghosts else [])
    return seq + ["residual"]


@pytest.mark.parametrize("wls,restrict,ghosts,n", [(57000, 0, 9000, 13), (0, 0, 400, 11), (900, 4, 100, 16), (0, 3, 0, 13),
                                                   (12, 0, 0, 10)])
def test_launches_of_a_step(wls, restrict, ghosts, n):
    cnt = dict(n_wls_requests=wls, n_restrict_requests=restrict, n_ghost=ghosts)
    assert bench.launches_per_step(cnt) == len(_sequence(wls, restrict, ghosts)) == n
