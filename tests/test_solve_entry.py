"""The entry point of the shifted solves and coefficients.  Its grid is sized
by the SMs, so it may be far larger than the partition: nothing in it may read
a table with an entry per block of the partition."""
import os
import re

import numpy as np
import pytest

from gpumatfun_gb300 import Engine, params, workloads
from oracle import fab

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpumatfun_gb300", "csrc")


def body(source: str, head: str) -> str:
    """Text of the function whose declaration contains head, to its closing brace."""
    at = source.index("{", re.search(head, source).end())
    depth = 0
    for i in range(at, len(source)):
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        if depth == 0:
            return re.sub(r"//[^\n]*", "", source[at:i])
    raise AssertionError("unbalanced braces")


@pytest.mark.parametrize("unit", ["kern_fp64.cu", "kern_mixed.cu"])
def test_reads_no_table_of_the_partition(unit):
    """The kernel registered for the solves, and what it calls, use
    no block tables (blk_*, prob_blk0, Grp, which reads both)."""
    kernel = re.search(r"case 1: return \(void\*\)(\w+)<", open(os.path.join(CSRC, unit)).read()).group(1)
    source = open(os.path.join(CSRC, "fab_kernel.cuh")).read()
    for head in (r"\b%s\(KParams kp\)" % kernel, r"\bclear_unwritten\(", r"\bphase_trisolve\(", r"\bphase_coef\("):
        assert not re.search(r"\bGrp\b|\bgroup_bar\b|\bblk_\w+|\bprob_blk0\b", body(source, head)), head


@pytest.mark.gpu
@pytest.mark.parametrize("R,C,m", [(1, 8, 5), (4, 200, 5), (2, 64, 3)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_one_block_of_rows_many_blocks_of_systems(engine_lib, precision, R, C, m):
    """A partition of one block, the three calls one by one; the engine's
    tolerances against the oracle, 1e-10 FP64 and 1e-6 mixed."""
    P = workloads.fd2d_problem(5, 2, m, C, [params.frac_exp(1e-3, 1.5)] * R, R=R, scale=36.0, seed=R, degree=1)
    e = Engine.from_problem(P, precision=precision, threads=64)
    e.build_subspace()
    e.lin_sys_solves()
    e.apply_V()
    x, info = e.get_solution(), e.info()
    e.delete()
    assert info["grid_blocks"] == 1
    want = fab.OracleEngine(A=P.A, U0=P.U, Q=P.Q, m=P.m, gamma=P.gamma, gs_re=P.gs_re, gs_im=P.gs_im, flam=P.flam,
                            wts=P.wts, shifts=P.shifts, col_scale=np.ones(R)).solve()
    assert np.linalg.norm(x - want) < (1e-10 if precision == "fp64" else 1e-6) * np.linalg.norm(want)
