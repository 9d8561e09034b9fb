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


def _shifted(t, by):
    """The same values in a dense tensor that starts `by` elements into its buffer."""
    buf = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)
    out = buf[by:].view(t.shape)
    out.copy_(t)
    assert out.is_contiguous() and out.data_ptr() % 16 != 0
    return out


@pytest.mark.parametrize("K,V", [(64, 64), (128, 64), (96, 32)])
@pytest.mark.parametrize("grads", [False, True])
def test_narrow_heads_at_odd_addresses(K, V, grads):
    """Heads of fewer than 128 columns: dense tensors that do not start on a 16-byte boundary are taken (they were padded into new ones
    once), with the results of aligned ones, gradients from odd addresses included."""
    from kda_b200 import chunk_kda
    d = {n: t.cuda() for n, t in make_inputs(1, 130, 2, K, V, torch.bfloat16, seed=3, h0_std=0.02, backward=True).items()}

    def run(shift):
        x = {n: (_shifted(d[n], by) if shift else d[n].clone()) for n, by in (("q", 1), ("k", 3), ("v", 4), ("g", 1), ("h0", 2), ("do", 5), ("dht", 1))}
        lv = [x[n].requires_grad_(grads) for n in ("q", "k", "v", "g")] + [d["beta"].clone().requires_grad_(grads), x["h0"].requires_grad_(grads)]
        o, ht = chunk_kda(*lv[:5], initial_state=lv[5], output_final_state=True)
        return [o, ht] + (list(torch.autograd.grad([o, ht], lv, [x["do"], x["dht"]])) if grads else [])

    for i, (a, b) in enumerate(zip(run(True), run(False))):
        assert torch.equal(a, b), i


def test_full_width_heads_at_odd_addresses_are_refused():
    from kda_b200 import _lib, chunk_kda
    d = _inputs(1, 70, 2, 128, 4)
    with pytest.raises(_lib.KdaError, match="align"):
        chunk_kda(_shifted(d["q"], 1), d["k"], d["v"], d["g"], d["beta"])


def test_bf16_gate_parameters_may_change_between_forward_and_backward():
    """The backward needs the float32 copies of A_log and dt_bias that the forward made; bf16 parameters may be updated in between."""
    from kda_b200 import chunk_kda
    d = _inputs(1, 100, 2, 128, 5)
    out = []
    for touch in (False, True):
        A, b = (torch.full((2,), 0.3, device="cuda").bfloat16().requires_grad_(True), torch.zeros(256, device="cuda").bfloat16().requires_grad_(True))
        o, _ = chunk_kda(d["q"], d["k"], d["v"], torch.sin(d["g"]), d["beta"], A_log=A, dt_bias=b, use_gate_in_kernel=True)
        if touch:
            with torch.no_grad():
                A.add_(1.0)
                b.sub_(1.0)
        out.append(torch.autograd.grad(o, [A, b], d["do"]))
    assert all(torch.equal(x, y) for x, y in zip(*out))
