"""The tensor-core step over its groupings of heads into stages (two stages are read out, appended and folded together, others one
after the other), and the step kernels on bf16 rows that do not lie on 8-byte boundaries, on a B200."""
import pytest
import torch

from test_step_gpu import DEV, _oracle_lockstep

import statequant_b200 as sq
from statequant_b200.kernels import SlotLayout

pytestmark = pytest.mark.gpu

# value and key heads: a CTA of one stage, of two, of three, and of five that go through a ring of four
GROUPS = [(2, 2), (4, 2), (3, 1), (5, 1)]


@pytest.mark.parametrize('fmt', [(4, 'k', 64), (8, 'k', 32), (4, 'v', 32), (8, 'v', 32), (8, 'k', 128)])
@pytest.mark.parametrize('hv,hk', GROUPS)
def test_tensor_core_step_over_head_groupings(fmt, hv, hk):
    """Two fold periods against the oracle, same bar as the other cases (fp32 sums in another order: 2e-5 of the largest output)."""
    from statequant_b200 import _cabi
    c = dict(kind='gdn', fmt=fmt, B=2, hv=hv, hk=hk, dk=128, dv=128, m=8, bb=8, seed=101)
    before = _cabi.path_counts()[4]
    _cabi.set_option('kernel_path', 4)
    try:
        st = _oracle_lockstep(c, T=19, act_dtype=torch.float32)
    finally:
        _cabi.set_option('kernel_path', 0)
    assert _cabi.path_counts()[4] - before == 19
    assert st['worst'] < 2e-5, st
    assert st['buf'] <= max(1, 1e-4 * st['nbuf']) and st['codes'] <= max(1, 1e-4 * st['ncodes']) and st['scal'] <= max(1, 1e-4 * st['ncodes']), st


@pytest.mark.parametrize('fmt', [(4, 'k', 64), (8, 'k', 32)])
def test_heads_of_64_rows_where_the_tensor_core_step_is_asked_for(fmt):
    """Gated DeltaNet heads of 64 rows run on the next kernel that takes them (grids beyond one wave come here by themselves)."""
    from statequant_b200 import _cabi
    _cabi.set_option('kernel_path', 4)
    try:
        st = _oracle_lockstep(dict(kind='gdn', fmt=fmt, B=2, hv=4, hk=2, dk=128, dv=64, m=8, bb=8, seed=102), T=19, act_dtype=torch.float32)
    finally:
        _cabi.set_option('kernel_path', 0)
    assert st['worst'] < 2e-5, st
    assert st['buf'] <= max(1, 1e-4 * st['nbuf']) and st['codes'] <= max(1, 1e-4 * st['ncodes']) and st['scal'] <= max(1, 1e-4 * st['ncodes']), st


@pytest.mark.parametrize('fmt,dk,dv,path', [((8, 'k', 32), 128, 128, 4), ((8, 'k', 32), 128, 128, 5), ((4, 'v', 32), 128, 128, 4),
                                            ((4, 'k', 64), 96, 192, 5), ('bf16', 128, 128, 5)])
@pytest.mark.parametrize('skew', [1, 2, 3])
def test_bf16_rows_off_the_8_byte_boundary(fmt, dk, dv, path, skew):
    """bf16 q and k whose rows start 2, 4 or 6 bytes off give, bit for bit, what aligned ones give, over a fold."""
    from statequant_b200 import _cabi
    hv, hk, B, T = 4, 2, 3, 9
    lay = SlotLayout(fmt if fmt == 'bf16' else sq.Quantizer(*fmt), hv, hk, dk, dv, m=8)
    gen = torch.Generator(device=DEV).manual_seed(5)
    r = lambda *s: torch.randn(*s, generator=gen, device=DEV)                             # noqa: E731
    idx = torch.arange(1, B + 1, dtype=torch.int32, device=DEV)
    S0 = r(B, hv, dv, dk)
    x = [(r(B, hk, dk).bfloat16(), r(B, hk, dk).bfloat16(), r(B, hv, dv).bfloat16(), -r(B, hv).abs() * 0.1, torch.sigmoid(r(B, hv))) for _ in range(T)]
    got = []
    _cabi.set_option('kernel_path', path)
    try:
        for off in (0, skew):
            blob = lay.alloc(B + 1, DEV)
            lay.write(lay.views(blob), idx, S0)
            out = torch.zeros(T, B, hv, dv, dtype=torch.bfloat16, device=DEV)
            for t, (q, k, v, g, beta) in enumerate(x):
                wide = torch.zeros(B, 2 * hk * dk + 4, dtype=torch.bfloat16, device=DEV)
                qw, kw = (wide[:, off + i * hk * dk:off + (i + 1) * hk * dk].unflatten(1, (hk, dk)) for i in (0, 1))
                qw.copy_(q)
                kw.copy_(k)
                assert qw.data_ptr() % 8 == 2 * off
                lay.step(lay.views(blob), idx, qw, kw, v, out[t], dk ** -0.5, g=g, beta=beta)
            got.append((out, blob))
    finally:
        _cabi.set_option('kernel_path', 0)
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
