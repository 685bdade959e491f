"""The split CG's prefetched, descending forms: the same bits as the form
without prefetches, at the edges of the 256-cell and 512-cell tiles, odd and
even sizes (one cell and two cells a thread in the update kernel), and the
register kernel's solution within the bound of ``test_resident_cg``."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

from tests.test_resident_cg import _ring, _solve  # noqa: E402

pytestmark = pytest.mark.gpu


# cells, block cap: one partial tile, whole tiles, one cell past them, several
# tiles a block and ragged last tiles
@pytest.mark.parametrize("n,cap", [(37, 148), (256, 1), (512, 1), (513, 2), (1024, 3), (7177, 3), (7178, 3), (80001, 0)])
@pytest.mark.parametrize("reach,long_every", [(3, 1), (5, 2)])
def test_prefetched_split_cg_keeps_the_bits(n, cap, reach, long_every):
    s, diag, val = _ring(n, reach, long_every)
    g = torch.Generator(device="cuda").manual_seed(5)
    rhs = torch.randn((1, n), dtype=torch.float64, device="cuda", generator=g)
    plain, st = _solve(s, diag, val, rhs, 25, cap)
    ref, st_ref = _solve(s, diag, val, rhs, 0, cap)
    assert st.status == st_ref.status == "ok"
    assert float((plain - ref).norm()) < 4e-11
    for variant in (27, 29, 30, 31):
        x, st_v = _solve(s, diag, val, rhs, variant, cap)
        assert torch.equal(x, plain) and st_v.iterations == st.iterations
