"""Forms of a call that an ordinary autograd function refuses or takes as a matter of course, and the native host path has to treat the same way."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from kda_b200.inputs import make_inputs

pytestmark = pytest.mark.gpu


def _inputs(B, T, H, D, seed, dtype=torch.bfloat16):
    return {n: t.cuda() for n, t in make_inputs(B, T, H, D, D, dtype, seed=seed, h0_std=0.02, backward=True).items()}


@pytest.mark.parametrize("which", ["q", "beta", "h0", "A_log"])
@pytest.mark.parametrize("grads", [False, True])
def test_forward_mode_tangents_are_refused_not_dropped(which, grads):
    from kda_b200 import chunk_kda
    d = _inputs(1, 70, 2, 128, 1)
    x = dict(q=d["q"], k=d["k"], v=d["v"], g=d["g"], beta=d["beta"], initial_state=d["h0"])
    kw = {}
    if which == "A_log":
        x["A_log"] = torch.zeros(2, device="cuda")
        kw = dict(use_gate_in_kernel=True)
    name = "initial_state" if which == "h0" else which
    if grads:
        x["v"] = x["v"].requires_grad_(True)
    with fwAD.dual_level():
        x[name] = fwAD.make_dual(x[name], torch.ones_like(x[name]))
        with pytest.raises(RuntimeError, match="jvp"):
            chunk_kda(**x, **kw)
    assert torch.isfinite(chunk_kda(d["q"], d["k"], d["v"], d["g"], d["beta"])[0].float()).all()
