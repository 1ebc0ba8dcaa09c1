"""The Rys polynomials (csrc/rys_poly.inc), both layouts, evaluated as the
kernels do below XMAX, against 60-digit golden nodes and weights (on the device,
and on both sides of XMAX: test_gpu_rys.py)."""
import json
import os
import re

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, '..', 'byteqc_b200', 'csrc')


def _array(text, name):
    m = re.search(r'\b%s\[\d+\] = \{(.*?)\};' % name, text, re.S)
    return np.array([float(v) for v in m.group(1).replace('\n', ' ').split(',') if v.strip()])


@pytest.fixture(scope='module')
def tables():
    text = open(os.path.join(CSRC, 'rys_tables.inc')).read() + open(os.path.join(CSRC, 'rys_poly.inc')).read()
    num = lambda name: int(re.search(r'#define %s (\d+)' % name, text).group(1))
    return {'ncoef': num('RYS_POLY_NCOEF'), 'per': num('RYS_PER_UNIT'),
            'xmax': _array(text, 'RYS_XMAX').astype(int), 'off': _array(text, 'RYS_POLY_OFFSET').astype(int),
            'rows': _array(text, 'RYS_POLY'), 'levels': _array(text, 'RYS_POLY_LM')}


@pytest.mark.parametrize('layout', ['rows', 'levels'])
def test_tables_match_golden(tables, layout):
    """Relative error at most 2e-15: the fit's remainder (below 5e-16 times a
    derivative of order one), the rounding of ten coefficients and of the
    argument's reduction to the interval."""
    golden = json.load(open(os.path.join(HERE, 'golden', 'rys_mpmath.json')))
    nc, per = tables['ncoef'], tables['per']
    seen = set()
    for g in golden:
        n, x = g['n'], float(g['x'])
        if x >= tables['xmax'][n]:
            continue
        nint = per * tables['xmax'][n]
        k = int(per * x)
        t = 2. * (per * x - k) - 1.
        tab = tables[layout][tables['off'][n]:tables['off'][n + 1]]
        if layout == 'rows':
            coef = tab.reshape(nint, nc, 2 * n)[k]
        else:
            coef = tab.reshape(nc, n, nint, 2)[:, :, k].reshape(nc, 2 * n)
        f = coef[nc - 1].copy()
        for c in coef[nc - 2::-1]:
            f = f * t + c
        ref = np.array([float(v) for v in g['r']] + [float(v) for v in g['w']])
        assert np.abs(f / ref - 1).max() < 2e-15, (n, x, np.abs(f / ref - 1).max())
        seen.add(n)
    assert seen == set(range(1, len(tables['xmax'])))
