"""sin and cos on the integer pipes and the item functions' shared operations: plain calls and batches give the
same bits, sin / cos within 2 ulp of libm for every kind of argument (its error and theirs are each below one),
and divisions the oracle's values at the edges of their divisors."""
import math

import numpy as np
import pytest

import helpers as H
import oracle as O
import ralgpu as R
from ralgpu import dtypes as D

pytestmark = pytest.mark.gpu


def _arguments(kind):
    rng = np.random.default_rng(len(kind))
    n = 20_011
    sign = rng.choice([-1.0, 1.0], n)
    if kind == "tiny":  # around the smallest argument with a series, subnormals, zeros
        x = np.ldexp(rng.uniform(1, 2, n), rng.integers(-40, 0, n))
        x[:64] = np.ldexp(1.0, np.arange(-1074, -1010))
        x[64:66] = 0.0
    elif kind == "quarter":  # next to the bounds of the reduction and to pi/4
        x = np.concatenate([np.nextafter(b, b + np.linspace(-1, 1, n // 4 + 1)) for b in (0.5, np.pi / 4, 2.0 ** -27, 1.0)])[:n]
    elif kind == "integers":
        x = rng.integers(0, 1 << 20, n).astype(np.float64)
    elif kind == "multiples":  # next to multiples of pi/2 of every size
        x = np.rint(np.ldexp(rng.uniform(0.5, 1, n), rng.integers(0, 50, n))) * (np.pi / 2)
    elif kind == "spread":
        x = np.ldexp(rng.uniform(1, 2, n), rng.integers(-1, 51, n))
    else:  # "far": 2^52 and more, infinities, NaN
        x = np.ldexp(rng.uniform(1, 2, n), rng.integers(50, 1023, n))
        x[:3] = [np.inf, -np.inf, np.nan]
    return x * sign


def _both(cols, query):
    """The query's outputs by a plain call and by a batch."""
    n = len(cols[0][1])
    frame = H.to_device(cols)
    plain = R.execute_project_plan(frame, query)
    pp = R.parse_project_plan([c[0] for c in cols], query)
    outs = [R.Column.empty(dt, n, with_valid=True) for dt in pp["evaluated_dtypes"]]
    b = R.Batch()
    b.add(outs, [frame[c] for c in pp["input_columns"]], pp["left"], pp["right"], pp["outputs"], pp["final_output_positions"],
          pp["operators"], pp["unary_operators"], pp["left_scalars"], pp["right_scalars"])
    b.prepare()
    b.run()
    for p, o in zip(plain, outs):
        np.testing.assert_array_equal(p.to_numpy().view(np.int64), o.to_numpy().view(np.int64))
    return [p.to_numpy() for p in plain]


@pytest.mark.parametrize("kind", ["tiny", "quarter", "integers", "multiples", "spread", "far"])
def test_sin_cos(kind):
    x = _arguments(kind)
    s, c = _both([(D.GDF_FLOAT64, x, None)], "LogicalProject(a=[SIN($0)], b=[COS($0)])")
    finite = np.isfinite(x)
    for got, fn in ((s, math.sin), (c, math.cos)):
        assert np.isnan(got[~finite]).all()
        exp = np.array([fn(v) for v in x[finite]])
        assert H.ulp_distance(got[finite], exp).max() <= H.ULP_TOL


def test_divisions():
    edge = np.array([0, 1, -1, 2, -2, 7, 1 << 16, (1 << 16) - 1, -(1 << 16), (1 << 32) - 1, 1 << 32, -(1 << 32) - 1,
                     (1 << 62) + 3, np.iinfo(np.int64).max, np.iinfo(np.int64).min], dtype=np.int64)
    rng = np.random.default_rng(3)
    a = np.concatenate([np.repeat(edge, len(edge)), rng.integers(-(1 << 62), 1 << 62, 5000)])
    b = np.concatenate([np.tile(edge, len(edge)), np.right_shift(rng.integers(-(1 << 62), 1 << 62, 5000), rng.integers(0, 62, 5000))])
    d = np.concatenate([np.repeat([0.0, -0.0, 1.0, -3.0, 5e-324, 1e-308, 1e308, np.inf, np.nan], 600), rng.standard_normal(a.size)])[:a.size]
    e = np.roll(d, 601)
    cols = [(D.GDF_INT64, a, None), (D.GDF_INT64, b, None), (D.GDF_FLOAT64, d, None), (D.GDF_FLOAT64, e, None)]
    query = "LogicalProject(q=[/($0, $1)], r=[MOD($0, $1)], f=[/($2, $3)])"
    got = _both(cols, query)
    exp = O.execute_project_plan(H.to_oracle(cols), query)
    for g, x in zip(got, exp):
        if g.dtype.kind == "f":
            np.testing.assert_array_equal(np.isnan(g), np.isnan(x.data))
            g, x = g[~np.isnan(g)], x.data[~np.isnan(x.data)]
            np.testing.assert_array_equal(g.view(np.int64), x.view(np.int64))
        else:
            np.testing.assert_array_equal(g, x.data)
