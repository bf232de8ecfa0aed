"""The split-precision kernels where slices still run as slices: small operators and contractions asked for
with slices get FP64 results from faster kernels, so the slice kernels are reached through batches,
prepared operators with few slices and applications above 20 GFLOP. Every test says that the split GEMM
was launched (or that it was not)."""
import numpy as np
import pytest

import mps_gb300 as mg
from mps_gb300 import dmrg as gd
from tests.helpers import relerr
from tests.test_gpu_batch import _oracle_apply
from tests.test_gpu_split import TOL

pytestmark = pytest.mark.gpu

SHAPES = [(64, 9, 3), (96, 11, 5), (48, 7, 7)]


def split_launches(ctx, f):
    ctx.set_timing(True)
    r = f()
    n = ctx.kernel_time("gemm_split")[1]
    ctx.set_timing(False)
    return r, n


def problems(ctx, shapes=SHAPES):
    return [gd.heff_problem(chi, 0.5, seed, ctx=ctx, ncharges=nq) for chi, nq, seed in shapes]


@pytest.mark.parametrize("S", [2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("tuning", [None, (64, 0, 0), (64, 1, 0), (128, 0, 0), (0, 0, 1)])
def test_batches(S, tuning):
    ctx = mg.Context(0)
    if tuning:
        mg.set_split_tuning(ctx, *tuning)
    ops = problems(ctx)
    B = mg.HeffBatch(ops, precision=S, graph=False)
    got, n = split_launches(ctx, lambda: B([o[0] for o in ops]))
    assert n == 2
    for g, shape in zip(got, SHAPES):
        assert relerr(g.to_flat(), _oracle_apply(*shape)) < 4 * TOL[S], shape


@pytest.mark.parametrize("S", [6, 7])
def test_batches_at_the_digit_bounds(S):
    """127.5/128 has the largest balanced digits; a constant operand takes every group sum to its bound."""
    ctx = mg.Context(0)
    ops = []
    for v, eL, eR, W1, W2 in problems(ctx, [(400, 7, 3), (64, 9, 5)]):
        ops.append(tuple(mg.fill_(mg.copy(t), 127.5 / 128) for t in (v, eL, eR)) + (W1, W2))
    B = mg.HeffBatch(ops, precision=S, graph=False)
    got, n = split_launches(ctx, lambda: B([o[0] for o in ops]))
    assert n == 2
    for g, op in zip(got, ops):
        assert relerr(g.to_flat(), mg.Heff2(*op, precision=0)(op[0]).to_flat()) < TOL[S]


@pytest.mark.parametrize("S", [2, 3, 4, 5])
def test_prepared_operators(S):
    """Two to four slices run as slices at every size, five from 4 GFLOP on (FP64 below)."""
    op = gd.heff_problem(64, 0.5, 1911, ncharges=9)
    H = mg.Heff2(*op, precision=S)
    got, n = split_launches(op[0].ctx, lambda: H(op[0]))
    assert n == (2 if S < 5 else 0)
    assert relerr(got.to_flat(), _oracle_apply(64, 9, 1911)) < 4 * TOL[S]


@pytest.mark.parametrize("S,batch", [(3, False), (4, False), (5, True), (7, True)])
def test_nan_input_propagates(S, batch):
    ctx = mg.Context(0)
    v, *rest = problems(ctx, SHAPES[:1])[0]
    bad = v.to_flat()
    bad[7] = np.nan
    vb = mg.from_flat(v.charge, v.space, bad, ctx)
    ok = mg.Heff2(v, *rest, precision=0)(v).to_flat()
    H = mg.HeffBatch([(v, *rest)], precision=S, graph=False) if batch else mg.Heff2(v, *rest, precision=S)
    out, n = split_launches(ctx, lambda: H([vb])[0] if batch else H(vb))
    assert n == 2
    out = out.to_flat()
    fin = np.isfinite(out)
    assert np.isnan(out).any() and fin.any()
    assert np.linalg.norm(out[fin] - ok[fin]) < 1e-4 * np.linalg.norm(ok[fin])


@pytest.mark.parametrize("S", [3, 4])
def test_host_buffers_above_the_limit(S):
    """chi = 2900, 23 GFLOP: the operator is prepared from environments that are still being uploaded."""
    (sv, sl, sr), flats = gd.heff_inputs_host(2900, 0.5, 1911, 25)
    D = gd.heff_problem(8, 0.5, 1911, ncharges=5)
    ctx = D[0].ctx
    dev = [mg.zeros(0, s) for s in (sv, sl, sr)] + [mg.copy(t) for t in D[3:]]
    host = [np.ascontiguousarray(f) for f in flats] + [t.to_flat() for t in D[3:]]
    assert mg.applymps2site_flops(*dev) > 2e10
    out = {}
    for s in (0, S):
        out[s] = np.zeros(dev[0].numel())
        _, n = split_launches(ctx, lambda: mg.applymps2site_host(*dev, host, out[s], precision=s))
        assert n == (2 if s else 0)
    assert relerr(out[S], out[0]) < 4 * TOL[S]
