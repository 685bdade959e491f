"""A slot's share of the GPU: its block caps are at most that share of the
blocks of the kernels it runs that fit on the GPU at once."""

from __future__ import annotations

from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

SMS = 148


@pytest.mark.parametrize("share", [0.01, 0.25, 0.5, 0.75])
# solver, cells, resident blocks an SM of the kernel it runs
@pytest.mark.parametrize("bicgstab,mixed,variant,n,per_sm", [
    (True, False, None, 16**3, 1), (True, True, None, 16**3, 1),
    (False, False, None, 16**3, 1), (False, False, None, 64**3, 1), (False, False, None, 110**3, 1),
    (False, True, None, 16**3, 4), (False, True, None, 48**3, 1), (False, True, None, 110**3, 2),
    (False, False, 0, 16**3, 4), (False, False, 2, 48**3, 2), (False, False, 10, 48**3, 1)])
def test_cap_is_a_share_of_the_coresident_blocks(share, bicgstab, mixed, variant, n, per_sm):
    from gridfoam_b200.serving.engine import block_cap

    s = SimpleNamespace(bicgstab=bicgstab, mixed=mixed, variant=variant)
    cap = block_cap(s, n, 3 if bicgstab else 1, 6, share, SMS, lambda ncomp, width, mixed: SMS)
    assert 1 <= cap <= max(1, share * SMS * per_sm)
    assert cap == max(1, int(share * SMS * per_sm))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["float64", "float32"])
def test_slots_with_half_the_gpu_stay_within_it(precision):
    from gridfoam_b200._lib import load
    from gridfoam_b200.serving import CavityRequest, ServingEngine
    from gridfoam_b200.serving.engine import _Slot

    eng = ServingEngine(max_slots=2, max_outer=4, gpu_share=0.5, inner_precision=precision)
    eng.prepare({16}, autotune=False)
    slot = _Slot(eng, CavityRequest(0, 16, 100.0, 1.0, 0.0), 0.0)
    torch.cuda.synchronize()
    caps = {name: s.block_cap for name, s in slot.algo.solvers.items()}
    assert caps["U"] <= 0.5 * load().gf_bicgstab_max_blocks(3, 6, int(precision == "float32"))
    # one block an SM is the least that any kernel has
    assert load().gf_bicgstab_max_blocks(3, 6, 0) >= eng.sms
    if precision == "float64":  # the default pressure CG runs one block an SM
        assert caps["p"] <= 0.5 * eng.sms


@pytest.mark.gpu
def test_bicgstab_block_query():
    from gridfoam_b200._lib import load

    lib = load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for ncomp in (1, 2, 3):
        for width in (6, 12):
            assert lib.gf_bicgstab_max_blocks(ncomp, width, 0) == sms  # 1024 threads of 64 registers
            assert lib.gf_bicgstab_max_blocks(ncomp, width, 1) in (sms, 2 * sms)
    assert lib.gf_bicgstab_max_blocks(4, 6, 0) == -1 and lib.gf_bicgstab_max_blocks(1, 0, 0) == -1
