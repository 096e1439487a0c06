"""A branch of a batch's graph runs each launch as the batch was tuned: the same tile and the same form of the dense
ops, though the branch has fewer lines than the rule for that form asks for.  The state after a step agrees with the
eager batch's to rounding (1e-11 of the largest coefficient: the forms differ by 1e-15 an operator)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_branches_keep_the_dense_form():
    from pypde_gb300.navier.fused import FusedBatch
    from pypde_gb300.navier.rbc2d import NavierStokes
    solvers = []
    for k, shape in enumerate([(81, 113), (113, 81), (81, 81), (113, 113), (81, 113), (113, 81)]):
        ns = NavierStokes(case="linear", shape=shape, ra=1e5, pr=1.0, dt=0.005, tsave=None)
        ns.set_temperature_noise(k, 0.1)
        solvers.append(ns)
    fb = FusedBatch(solvers, split=False)
    x0 = fb.state_arena.clone()
    fb.step_eager()
    ref = fb.state_arena.clone()
    forms = {(L["name"], L["key"]): (L["P"].tb, L["P"].nthreads, L["tc"]) for g in fb.launches for L in g}
    assert any(f[2] for f in forms.values())
    for idx in ([0], [1, 2]):
        for g in fb._subset(idx).launches:
            for L in g:
                assert (L["P"].tb, L["P"].nthreads, L["tc"]) == forms[(L["name"], L["key"])]
    fb.state_arena.copy_(x0)
    fb.capture(1, groups="shape")
    fb.state_arena.copy_(x0)
    fb.step()
    torch.cuda.synchronize()
    assert (fb.state_arena - ref).abs().max() <= 1e-11 * ref.abs().max()
