"""GPU parity of the float32 training path (token-recurrent forward and its exact reverse mode: two walks over the tokens and
32-token pieces between them, `kda_recurrent_train.cu`) against float64 autograd through the token-by-token oracle: max-normalised error <= 1e-4 for
o, the final state and every gradient (the fp32-mode bar)."""
import numpy as np
import pytest
import torch

from kda_b200.inputs import make_inputs
from oracle.kda_oracle import max_norm_err, recurrent_kda_grads

pytestmark = pytest.mark.gpu
NAMES = ("o", "ht", "dq", "dk", "dv", "dg", "dbeta", "dh0")
TOL = 1e-4


def _run(d, cu=None, scale=None, l2=False, with_h0=True, transpose=False):
    from kda_b200 import chunk_kda
    lv = {n: d[n].cuda().requires_grad_(True) for n in ("q", "k", "v", "g", "beta")}
    h0 = None
    if with_h0 and d["h0"] is not None:
        h0 = d["h0"].cuda()
        if transpose:
            h0 = h0.transpose(-1, -2).contiguous()
        h0.requires_grad_(True)
    o, ht = chunk_kda(lv["q"], lv["k"], lv["v"], lv["g"], lv["beta"], scale=scale, initial_state=h0, output_final_state=True,
                      use_qk_l2norm_in_kernel=l2, cu_seqlens=None if cu is None else cu.cuda(), transpose_state_layout=transpose)
    assert o.dtype == torch.float32 and ht.dtype == torch.float32
    dht = d["dht"].cuda()
    torch.autograd.backward([o, ht], [d["do"].cuda(), dht.transpose(-1, -2).contiguous() if transpose else dht])
    un = (lambda t: t.transpose(-1, -2)) if transpose else (lambda t: t)
    return dict(o=o.detach(), ht=un(ht.detach()), dq=lv["q"].grad, dk=lv["k"].grad, dv=lv["v"].grad, dg=lv["g"].grad,
                dbeta=lv["beta"].grad, dh0=None if h0 is None else un(h0.grad))


def _check(got, ref):
    for n in NAMES:
        if ref[n] is None or got[n] is None:
            continue
        assert torch.isfinite(got[n]).all(), n
        e = max_norm_err(got[n], ref[n])
        assert e <= TOL, f"{n}: max-normalised error {e:.3e}"


@pytest.mark.parametrize("T", [1, 63, 64, 65, 200])
def test_fp32_backward_lengths(T):
    d = make_inputs(2, T, 2, 128, 128, torch.float32, seed=300 + T, h0_std=0.1, backward=True)
    ref = recurrent_kda_grads(d["q"], d["k"], d["v"], d["g"], d["beta"], d["do"], d["dht"], initial_state=d["h0"])
    _check(_run(d), ref)


@pytest.mark.parametrize("K,V", [(32, 32), (64, 64), (64, 128), (128, 32), (32, 64)])
def test_fp32_backward_head_sizes(K, V):
    d = make_inputs(1, 150, 3, K, V, torch.float32, seed=400 + K + V, h0_std=0.1, backward=True)
    ref = recurrent_kda_grads(d["q"], d["k"], d["v"], d["g"], d["beta"], d["do"], d["dht"], initial_state=d["h0"])
    _check(_run(d), ref)


def test_fp32_backward_l2norm_scale_no_h0():
    d = make_inputs(1, 130, 2, 64, 64, torch.float32, seed=41, backward=True)
    d["q"], d["k"] = d["q"] * 2.5, d["k"] * 0.4
    ref = recurrent_kda_grads(d["q"], d["k"], d["v"], d["g"], d["beta"], d["do"], d["dht"], scale=0.2, use_qk_l2norm=True)
    _check(_run(d, scale=0.2, l2=True, with_h0=False), ref)


def test_fp32_backward_packed_with_an_empty_sequence_and_transposed_states():
    lens = [70, 0, 1, 129]
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32)
    d = make_inputs(1, sum(lens), 2, 128, 128, torch.float32, seed=42, h0_std=0.1, n_states=len(lens), backward=True)
    ref = recurrent_kda_grads(d["q"], d["k"], d["v"], d["g"], d["beta"], d["do"], d["dht"], initial_state=d["h0"],
                              cu_seqlens=cu, use_qk_l2norm=True)
    got = _run(d, cu=cu, l2=True, transpose=True)
    _check(got, ref)
    assert torch.equal(got["dh0"][1].cpu(), d["dht"][1])      # the empty sequence hands its state gradient through


def test_fp32_backward_grouped_value_heads():
    """q, k with one head shared by two value heads: dq, dk are the sums over the group."""
    d = make_inputs(1, 100, 2, 64, 64, torch.float32, seed=43, h0_std=0.1, backward=True)
    d["q"], d["k"] = d["q"][:, :, :1].contiguous(), d["k"][:, :, :1].contiguous()
    rep = lambda t: t.expand(-1, -1, 2, -1)      # noqa: E731
    lq, lk = d["q"].double().requires_grad_(True), d["k"].double().requires_grad_(True)
    from oracle.kda_oracle import recurrent_kda
    rest = [d[n].double().requires_grad_(True) for n in ("v", "g", "beta")]
    h0 = d["h0"].double().requires_grad_(True)
    o, ht = recurrent_kda(rep(lq), rep(lk), *rest, initial_state=h0, output_final_state=True)
    gr = torch.autograd.grad([o, ht], [lq, lk] + rest + [h0], [d["do"].double(), d["dht"].double()])
    ref = dict(o=o.detach(), ht=ht.detach(), dq=gr[0], dk=gr[1], dv=gr[2], dg=gr[3], dbeta=gr[4], dh0=gr[5])
    _check(_run(d), ref)


def test_fp32_backward_is_deterministic():
    d = make_inputs(2, 100, 2, 128, 128, torch.float32, seed=44, h0_std=0.1, backward=True)
    a, b = _run(d), _run(d)
    for n in NAMES:
        assert torch.equal(a[n], b[n]), n


# longer calls: several hundred tokens, an empty sequence between others
@pytest.mark.parametrize("lens,K,V,l2,transpose", [([256], 128, 128, False, False), ([257], 128, 128, True, False), ([303], 64, 128, False, True),
                                                   ([64, 0, 1, 63, 145], 128, 128, True, True)])
def test_fp32_training_of_longer_calls(lens, K, V, l2, transpose):
    N = len(lens)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32) if N > 1 else None
    d = make_inputs(1, sum(lens), 3, K, V, torch.float32, seed=500 + sum(lens), h0_std=0.1, n_states=N, backward=True)
    if l2:
        d["q"], d["k"] = d["q"] * 2.5, d["k"] * 0.4
    ref = recurrent_kda_grads(d["q"], d["k"], d["v"], d["g"], d["beta"], d["do"], d["dht"], initial_state=d["h0"], cu_seqlens=cu,
                              use_qk_l2norm=l2)
    _check(_run(d, cu=cu, l2=l2, transpose=transpose), ref)


def test_fp32_training_grouped_value_heads_longer():
    from oracle.kda_oracle import recurrent_kda
    d = make_inputs(2, 150, 4, 128, 128, torch.float32, seed=47, h0_std=0.1, backward=True)
    d["q"], d["k"] = d["q"][:, :, :2].contiguous(), d["k"][:, :, :2].contiguous()
    lv = [d[n].double().requires_grad_(True) for n in ("q", "k", "v", "g", "beta", "h0")]
    two = lambda t: t.repeat_interleave(2, dim=2)      # noqa: E731
    o, ht = recurrent_kda(two(lv[0]), two(lv[1]), *lv[2:5], initial_state=lv[5], output_final_state=True)
    gr = torch.autograd.grad([o, ht], lv, [d["do"].double(), d["dht"].double()])
    _check(_run(d), dict(o=o.detach(), ht=ht.detach(), dq=gr[0], dk=gr[1], dv=gr[2], dg=gr[3], dbeta=gr[4], dh0=gr[5]))


@pytest.mark.parametrize("K,V", [(40, 24), (96, 64), (128, 256)])
def test_fp32_gradients_of_other_head_sizes_are_refused(K, V):
    from kda_b200 import chunk_kda
    d = make_inputs(1, 300, 2, K, V, torch.float32, seed=48)
    lv = [d[n].cuda().requires_grad_(True) for n in ("q", "k", "v", "g", "beta")]
    with pytest.raises(NotImplementedError, match="float32 gradients need K, V"):
        chunk_kda(*lv)


@pytest.mark.parametrize("B,T,H,D", [(2, 512, 4, 64), (1, 512, 4, 128)])
def test_fp32_layer_gradients_are_float32_accurate(B, T, H, D):
    """The layer's call (raw gate, beta logits, L2 norm) in float32.  The gradients of A_log and dt_bias sum the gate gradients of all tokens, large
    terms of either sign: whatever a backward loses in dg shows there many times over.  Against float64 autograd through the token-by-token
    oracle, 2-norm: 1e-5 (products and sums in float32, a few hundred terms: 2^-24 sqrt(B T) = 2e-6, gate functions 1e-6; measured 1e-6)."""
    import torch.nn.functional as F
    from kda_b200 import chunk_kda
    from oracle.kda_oracle import recurrent_kda
    gen = torch.Generator().manual_seed(49)
    rn = lambda *s: torch.randn(*s, generator=gen)      # noqa: E731
    x = dict(q=rn(B, T, H, D), k=rn(B, T, H, D), v=rn(B, T, H, D), g=rn(B, T, H, D), beta=rn(B, T, H),
             A_log=torch.log(1.0 + 15.0 * torch.rand(H, generator=gen)), dt_bias=rn(H * D))
    up = rn(B, T, H, D)
    lv = {n: t.cuda().requires_grad_(True) for n, t in x.items()}
    o, _ = chunk_kda(**lv, use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True)
    got = dict(zip(lv, torch.autograd.grad(o, list(lv.values()), up.cuda())))
    r = {n: t.cuda().double().requires_grad_(True) for n, t in x.items()}
    g = -torch.exp(r["A_log"]).view(1, 1, H, 1) * F.softplus(r["g"] + r["dt_bias"].view(1, 1, H, D), threshold=1e9)
    ro, _ = recurrent_kda(r["q"], r["k"], r["v"], g, torch.sigmoid(r["beta"]), use_qk_l2norm=True)
    ref = dict(zip(r, torch.autograd.grad(ro, list(r.values()), up.cuda().double())))
    for n in x:
        e = float((got[n].double() - ref[n]).norm() / ref[n].norm())
        assert e <= 1e-5, f"d_{n}: relative error {e:.2e}"


def test_fp32_gradients_at_odd_addresses():
    """Incoming gradients that do not start on a 16-byte boundary (views into a larger buffer) give the results of aligned ones."""
    from kda_b200 import chunk_kda
    d = {n: t.cuda() for n, t in make_inputs(1, 70, 2, 64, 64, torch.float32, seed=50, h0_std=0.1, backward=True).items()}
    lv = [d[n].requires_grad_(True) for n in ("q", "k", "v", "g", "beta", "h0")]
    out = []
    for shift in (0, 1):
        ups = []
        for n in ("do", "dht"):
            buf = torch.zeros(d[n].numel() + shift, device="cuda")
            ups.append(buf[shift:].view(d[n].shape).copy_(d[n]))
        o, ht = chunk_kda(*lv[:5], initial_state=lv[5], output_final_state=True)
        out.append(torch.autograd.grad([o, ht], lv, ups))
    assert all(torch.equal(a, b) for a, b in zip(*out))


def _errors(got, ref, bound):
    from oracle.kda_oracle import rel_l2_err
    for n in NAMES:
        if ref[n] is not None and got[n] is not None:
            e = rel_l2_err(got[n], ref[n])
            assert e <= bound, f"{n}: relative error {e:.2e}"


# 2-norm bound of the tests below: float32 steps, each rounding independent (2^-24 = 6e-8), over sums of up to 128 products and a few dozen
# dependent tokens: 6e-8 sqrt(64) = 5e-7; measured 1.2e-7.
EXACT = 5e-7


@pytest.mark.parametrize("T", [7, 8, 9, 31, 32, 33, 40, 61])
def test_fp32_training_at_the_edges_of_stages_and_kept_states(T):
    """The walks stage eight tokens at a time and keep a state every 32; the middle works on four tokens at a time, with the states between them in tensor memory."""
    d = make_inputs(2, T, 2, 128, 128, torch.float32, seed=600 + T, h0_std=0.1, backward=True)
    ref = recurrent_kda_grads(d["q"], d["k"], d["v"], d["g"], d["beta"], d["do"], d["dht"], initial_state=d["h0"])
    _errors(_run(d), ref, EXACT)


def _wide_batch(V, H):
    """Sequences that make enough (sequence, head) units for the walks with 32 columns a warp: units * V / 32 > 4 warps per SM."""
    return 4 * torch.cuda.get_device_properties(0).multi_processor_count * 32 // (V * H) + 1


@pytest.mark.parametrize("K,V", [(32, 32), (32, 64), (32, 128), (64, 32), (64, 64), (64, 128), (128, 32), (128, 64), (128, 128)])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("l2", [True, False])
def test_fp32_training_of_both_walks(K, V, wide, l2):
    """Many and few (sequence, head) units; with normalised rows (dq, dk through the last kernel) and without (dq, dk straight from the middle)."""
    H = 4
    B = _wide_batch(V, H) if wide else 1
    d = make_inputs(B, 37, H, K, V, torch.float32, seed=700 + K + V, h0_std=0.1, backward=True)
    ref = recurrent_kda_grads(*(d[n].cuda() for n in ("q", "k", "v", "g", "beta", "do", "dht")), initial_state=d["h0"].cuda(), use_qk_l2norm=l2)
    _errors(_run(d, l2=l2), ref, EXACT)


@pytest.mark.parametrize("l2", [False, True])
@pytest.mark.parametrize("HQ", [4, 2])
@pytest.mark.parametrize("kept", [True, False])
def test_fp32_training_of_many_uneven_sequences(l2, HQ, kept, monkeypatch):
    """The walks with 32 columns a warp over packed sequences of 0 to 70 tokens, with and without grouped value heads, from what the forward kept and
    replayed."""
    from kda_b200 import chunk_kda, ops
    monkeypatch.setattr(ops, "_keep_limit", lambda index: (1 << 30) if kept else 0)
    H, D = 4, 128
    lens = [(0, 1, 37, 32, 5, 70, 33)[i % 7] for i in range(_wide_batch(D, H))]
    tokens, N = sum(lens), len(lens)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    d = {n: t.cuda() for n, t in make_inputs(1, tokens, H, D, D, torch.float32, seed=58 + HQ, h0_std=0.1, n_states=N, backward=True).items()
         if t is not None}
    d["q"], d["k"] = (d[n][:, :, :HQ].contiguous() for n in ("q", "k"))
    each = lambda t: t.repeat_interleave(H // HQ, 2)      # noqa: E731
    ref = recurrent_kda_grads(each(d["q"]), each(d["k"]), *(d[n] for n in ("v", "g", "beta", "do", "dht")), initial_state=d["h0"], cu_seqlens=cu,
                              use_qk_l2norm=l2)
    for n in ("dq", "dk"):
        ref[n] = ref[n].view(1, tokens, HQ, H // HQ, D).sum(3)
    lv = [d[n].requires_grad_(True) for n in ("q", "k", "v", "g", "beta", "h0")]
    o, ht = chunk_kda(*lv[:5], initial_state=lv[5], output_final_state=True, cu_seqlens=cu, use_qk_l2norm_in_kernel=l2)
    assert bool(ops._kept) == kept
    grads = torch.autograd.grad([o, ht], lv, [d["do"], d["dht"]])
    _errors(dict(zip(NAMES, (o.detach(), ht.detach(), *grads))), ref, EXACT)


def test_recurrent_bwd_takes_q_k_g_at_odd_addresses():
    """The C entry asks no alignment of q, k and g: views one float into a buffer give the same bits."""
    import ctypes as C
    from kda_b200 import _lib
    lib = _lib.load()
    T, H, D = 70, 2, 64
    d = {n: t.cuda() for n, t in make_inputs(1, T, H, D, D, torch.float32, seed=51, backward=True).items() if t is not None}
    p = lambda t: C.c_void_p(t.data_ptr())      # noqa: E731
    out = []
    for shift in (0, 1):
        x = {}
        for n in ("q", "k", "g"):
            buf = torch.zeros(d[n].numel() + shift, device="cuda")
            x[n] = buf[shift:].view(d[n].shape).copy_(d[n])
        r = {n: torch.empty_like(d[n[1:]]) for n in ("dq", "dk", "dv", "dg", "dbeta")}
        ws = torch.empty(lib.kda_recurrent_bwd_workspace_bytes(T, 1, H, D, D), dtype=torch.uint8, device="cuda")
        a = _lib.RecurrentBwdArgs(q=p(x["q"]), k=p(x["k"]), v=p(d["v"]), g=p(x["g"]), beta=p(d["beta"]), d_o=p(d["do"]), workspace=p(ws),
                                  workspace_bytes=ws.numel(), tokens=T, N=1, T=T, H=H, K=D, V=D, HQ=H, io_dtype=_lib.KDA_FP32, use_qk_l2norm=1,
                                  scale=D ** -0.5, **{n: p(t) for n, t in r.items()})
        _lib.check(lib.kda_recurrent_bwd(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "kda_recurrent_bwd")
        torch.cuda.synchronize()
        out.append(r)
    assert all(torch.equal(out[0][n], out[1][n]) for n in out[0])


def test_fp32_backward_twice_through_one_forward():
    """What the forward keeps is only read: a second backward through the same graph gives the same bits."""
    from kda_b200 import chunk_kda
    d = {n: t.cuda() for n, t in make_inputs(1, 100, 2, 128, 128, torch.float32, seed=52, backward=True).items() if t is not None}
    lv = [d[n].requires_grad_(True) for n in ("q", "k", "v", "g", "beta")]
    o, _ = chunk_kda(*lv)
    a = torch.autograd.grad(o, lv, d["do"], retain_graph=True)
    b = torch.autograd.grad(o, lv, d["do"])
    assert all(torch.equal(x, y) for x, y in zip(a, b))


def _backward_us(B, T, H):
    from kda_b200 import chunk_kda
    d = {n: t.cuda() for n, t in make_inputs(B, T, H, 128, 128, torch.float32, seed=53, backward=True).items() if t is not None}
    lv = [d[n].requires_grad_(True) for n in ("q", "k", "v", "g", "beta")]
    o, _ = chunk_kda(*lv)
    times = []
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        torch.autograd.grad(o, lv, d["do"], retain_graph=True)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 1e3)
    return min(times)


def test_fp32_backward_of_short_sequences_does_not_cost_32_tokens():
    """The middle works on pieces of 32 tokens and stops behind the last token of a shorter one.  4,096 states of one token against the same
    of 32: 424 of 1,742 us (the states' traffic remains); with every piece walked to its end 1,231 of 1,832."""
    assert _backward_us(128, 1, 32) < 0.5 * _backward_us(128, 32, 32)


@pytest.mark.parametrize("l2,states", [(False, True), (True, False)])
def test_fp32_training_calls_keep_no_more_than_their_share(l2, states, monkeypatch):
    """Between forward and backward float32 calls keep intermediates up to a bound for all of them together; a call beyond it holds no memory but its
    results, unless it is asked to (`disable_recompute`).  What one call kept is given back with its backward.  The same bits either way."""
    from kda_b200 import chunk_kda, ops
    d = {n: t.cuda() for n, t in make_inputs(2, 333, 4, 128, 128, torch.float32, seed=54, h0_std=0.1, backward=True).items() if t is not None}
    lv = [d[n].requires_grad_(True) for n in ("q", "k", "v", "g", "beta", "h0")[:6 if states else 5]]
    one = 2 * (333 // 32) * 4 * 65536 + 2 * 333 * 4 * 512      # a state per 32 tokens and r, at least
    monkeypatch.setattr(ops, "_keep_limit", lambda index: 3 * one)

    def forward(**kw):
        before = torch.cuda.memory_allocated()
        o, ht = chunk_kda(*lv[:5], initial_state=lv[5] if states else None, output_final_state=states, use_qk_l2norm_in_kernel=l2, **kw)
        kept = torch.cuda.memory_allocated() - before - o.numel() * 4 - (ht.numel() * 4 if states else 0)
        return [o, ht][:1 + states], kept

    def backward(r, **kw):
        return [*r, *torch.autograd.grad(r, lv, [d["do"], d["dht"]][:1 + states], **kw)]

    calls = [forward() for _ in range(4)]                       # two have room, then none, then one that is asked to
    calls.append(forward(disable_recompute=True))
    assert [k >= one for _, k in calls] == [True, True, False, False, True]
    assert all(k < 4096 for _, k in calls[2:4])
    got = [backward(r, retain_graph=i == 0) for i, (r, _) in enumerate(calls)]
    assert forward()[1] >= one                                  # (its graph goes at once)
    assert [forward()[1] >= one for _ in range(3)] == [True] * 3
    got.append(backward(calls[0][0]))
    assert not ops._kept
    o, _ = chunk_kda(*(t[:1, :48] for t in lv[:5]))            # a short call replays
    assert o.requires_grad and not ops._kept
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.parametrize("lens", [[1, 1, 1], [32, 64, 31, 33], [3, 0, 96, 5, 32, 40]])
@pytest.mark.parametrize("over", ["nothing", "d_ht", "h0"])
@pytest.mark.parametrize("saved", [False, True])
def test_fp32_backward_scratch_bits_margins_and_states_in_place(lens, over, saved):
    """kda_recurrent_bwd_scratch with exactly the scratch it asks for, between sentinel margins, after either forward; dh0 over d_ht or h0, which the
    last kernel reads after the walk has written dh0.  The bits of the operator's autograd path, pieces that end on and off a multiple of 32."""
    import ctypes as C
    from _abi import guarded_like
    from kda_b200 import _lib, chunk_kda
    lib = _lib.load()
    tokens, N, H, D = sum(lens), len(lens), 2, 128
    d = make_inputs(1, tokens, H, D, D, torch.float32, seed=55 + tokens, h0_std=0.1, n_states=N, backward=True)
    d = {n: t.cuda().contiguous() for n, t in d.items()}
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    lv = {n: d[n].clone().requires_grad_(True) for n in ("q", "k", "v", "g", "beta", "h0")}
    o, ht = chunk_kda(*(lv[n] for n in ("q", "k", "v", "g", "beta")), initial_state=lv["h0"], output_final_state=True, cu_seqlens=cu,
                      use_qk_l2norm_in_kernel=True)
    torch.autograd.backward([o, ht], [d["do"], d["dht"]])
    guards, out = [], {}
    for n in ("q", "k", "v", "g", "beta", "h0"):
        g, out[n] = guarded_like(tuple(d[n].shape), torch.float32)
        guards.append((n, g))
    h0, dht = d["h0"], d["dht"]
    if over == "d_ht":
        dht = out["h0"].copy_(dht)
    elif over == "h0":
        h0 = out["h0"].copy_(h0)
    p = lambda t: C.c_void_p(t.data_ptr())      # noqa: E731
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    sizes = dict(tokens=tokens, N=N, T=0, H=H, K=D, V=D, HQ=H, io_dtype=_lib.KDA_FP32, use_qk_l2norm=1, scale=D ** -0.5)
    kept = None
    if saved:
        sg, kept = guarded_like((lib.kda_recurrent_saved_bytes(tokens, N, H, D, D),), torch.uint8)
        og, o2 = guarded_like(tuple(d["v"].shape), torch.float32)
        guards += [("saved", sg), ("o", og)]
        f = _lib.RecurrentArgs(q=p(d["q"]), k=p(d["k"]), v=p(d["v"]), g=p(d["g"]), beta=p(d["beta"]), h0=p(h0), o=p(o2), cu_seqlens=p(cu), **sizes)
        _lib.check(lib.kda_recurrent_train_fwd(C.byref(f), p(kept), kept.numel(), st), "kda_recurrent_train_fwd")
        assert torch.equal(o2, o)
    a = _lib.RecurrentBwdArgs(q=p(d["q"]), k=p(d["k"]), v=p(d["v"]), g=p(d["g"]), beta=p(d["beta"]), h0=p(h0), cu_seqlens=p(cu), d_o=p(d["do"]),
                              d_ht=p(dht), dq=p(out["q"]), dk=p(out["k"]), dv=p(out["v"]), dg=p(out["g"]), dbeta=p(out["beta"]), dh0=p(out["h0"]),
                              **sizes)
    wg, ws = guarded_like((lib.kda_recurrent_bwd_scratch_bytes(C.byref(a), saved, 1),), torch.uint8)
    a.workspace, a.workspace_bytes = p(ws), ws.numel()
    _lib.check(lib.kda_recurrent_bwd_scratch(C.byref(a), p(kept) if saved else None, kept.numel() if saved else 0, st), "kda_recurrent_bwd_scratch")
    torch.cuda.synchronize()
    for n, g in [*guards, ("scratch", wg)]:
        assert g.margins_intact(), n
    for n in out:
        assert torch.equal(out[n], lv[n].grad), n


@pytest.mark.parametrize("K,V,HQ,H,l2,lens", [(128, 128, 5, 5, False, [70, 32, 5]), (64, 128, 2, 6, False, [33, 64]), (128, 32, 3, 3, True, [200]),
                                              (128, 128, 3, 6, True, [1, 96, 40])])
@pytest.mark.parametrize("saved", [False, True])
def test_fp32_backward_over_groups_of_heads(K, V, HQ, H, l2, lens, saved):
    """A scratch that does not hold all heads: they are worked on in groups (of one q/k head, and of as many as two thirds of the scratch hold),
    between sentinel margins; the bits of the whole call."""
    import ctypes as C
    from _abi import guarded_like
    from kda_b200 import _lib
    lib = _lib.load()
    tokens, N = sum(lens), len(lens)
    d = make_inputs(1, tokens, H, K, V, torch.float32, seed=56 + tokens, h0_std=0.1, n_states=N, backward=True)
    d = {n: t.cuda().contiguous() for n, t in d.items()}
    d["q"], d["k"] = (d[n][:, :, :HQ].contiguous() for n in ("q", "k"))
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())      # noqa: E731
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    sizes = dict(tokens=tokens, N=N, T=0, H=H, K=K, V=V, HQ=HQ, io_dtype=_lib.KDA_FP32, use_qk_l2norm=int(l2), scale=K ** -0.5)
    inputs = dict(q=p(d["q"]), k=p(d["k"]), v=p(d["v"]), g=p(d["g"]), beta=p(d["beta"]), h0=p(d["h0"]), cu_seqlens=p(cu))
    kept, kept_bytes = None, 0
    if saved:
        kept = torch.empty(lib.kda_recurrent_saved_bytes(tokens, N, H, K, V), dtype=torch.uint8, device="cuda")
        kept_bytes, o = kept.numel(), torch.empty_like(d["v"])
        f = _lib.RecurrentArgs(**inputs, o=p(o), **sizes)
        _lib.check(lib.kda_recurrent_train_fwd(C.byref(f), p(kept), kept_bytes, st), "kda_recurrent_train_fwd")
    got = []
    for part in (1.0, 2 / 3, 1 / HQ):
        guards, out = [], {}
        for n in ("q", "k", "v", "g", "beta", "h0"):
            g, out[n] = guarded_like(tuple(d[n].shape), torch.float32)
            guards.append((n, g))
        a = _lib.RecurrentBwdArgs(**inputs, d_o=p(d["do"]), d_ht=p(d["dht"]), dq=p(out["q"]), dk=p(out["k"]), dv=p(out["v"]), dg=p(out["g"]),
                                  dbeta=p(out["beta"]), dh0=p(out["h0"]), **sizes)
        whole = lib.kda_recurrent_bwd_scratch_bytes(C.byref(a), saved, 1)
        size = whole if part == 1 else int(part * whole) + 7 * 256      # (each of the buffers is rounded up to 256 bytes)
        wg, ws = guarded_like((size,), torch.uint8)
        a.workspace, a.workspace_bytes = p(ws), size
        _lib.check(lib.kda_recurrent_bwd_scratch(C.byref(a), p(kept) if saved else None, kept_bytes, st), "kda_recurrent_bwd_scratch")
        torch.cuda.synchronize()
        for n, g in [*guards, ("scratch", wg)]:
            assert g.margins_intact(), n
        got.append(out)
    for n in got[0]:
        assert torch.equal(got[0][n], got[1][n]) and torch.equal(got[0][n], got[2][n]), n
    ref = recurrent_kda_grads(d["q"].repeat_interleave(H // HQ, 2), d["k"].repeat_interleave(H // HQ, 2), *(d[n] for n in ("v", "g", "beta", "do", "dht")),
                              initial_state=d["h0"], cu_seqlens=cu, use_qk_l2norm=l2)
    assert max_norm_err(got[0]["v"], ref["dv"]) <= TOL and max_norm_err(got[0]["g"], ref["dg"]) <= TOL
    for n in ("q", "k"):
        assert max_norm_err(got[0][n], ref["d" + n].view(1, tokens, HQ, H // HQ, K).sum(3)) <= TOL, n


@pytest.mark.parametrize("kept", [True, False])
def test_fp32_backward_takes_the_memory_that_is_there(kept, monkeypatch):
    """An allocator that has no room for the scratch of all heads at once (68 MB here, 152 with the replay): the call makes do with a part, same bits."""
    from kda_b200 import chunk_kda, ops
    if not kept:
        monkeypatch.setattr(ops, "_keep_limit", lambda index: 0)
    d = {n: t.cuda() for n, t in make_inputs(1, 4096, 8, 128, 128, torch.float32, seed=57, backward=True).items() if t is not None}
    lv = [d[n].requires_grad_(True) for n in ("q", "k", "v", "g", "beta")]
    first = torch.autograd.grad(chunk_kda(*lv)[0], lv, d["do"])
    o, _ = chunk_kda(*lv)
    asked, real = [], torch.empty

    def empty(*size, **kw):
        if kw.get("dtype") == torch.uint8:
            asked.append(size[0])
            if size[0] > 25 << 20:
                raise torch.OutOfMemoryError("no room")
        return real(*size, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    second = torch.autograd.grad(o, lv, d["do"])
    row = 4096 * (2048 + 32 + (0 if kept else 2048 + 512))
    assert asked == [n * row for n in ((8, 4, 2) if kept else (8, 4, 2, 1))]
    assert all(torch.equal(a, b) for a, b in zip(first, second))


@pytest.mark.parametrize("K,V,l2", [(128, 128, False), (64, 128, True), (32, 32, False)])
def test_fp32_training_of_packed_sequences_gives_each_one_its_own_bits(K, V, l2):
    """A batch that takes the walks with 32 columns a warp, and its sequences alone, which take those with 16: o, states and gradients are equal."""
    H = 4
    lens = [(70, 1, 37, 32, 9)[i % 5] for i in range(_wide_batch(V, H))]
    d = {n: t.cuda() for n, t in make_inputs(1, sum(lens), H, K, V, torch.float32, seed=59, h0_std=0.1, n_states=len(lens), backward=True).items()
         if t is not None}
    starts = np.concatenate([[0], np.cumsum(lens)])
    packed = _run({n: t.clone() for n, t in d.items()}, cu=torch.tensor(starts, dtype=torch.int32), l2=l2)
    for i in (0, 1, 2, 3, 4, len(lens) - 1):
        s, e = int(starts[i]), int(starts[i + 1])
        alone = _run({n: (t[i:i + 1] if n in ("h0", "dht") else t[:, s:e]).clone() for n, t in d.items()}, l2=l2)
        for n in NAMES:
            assert torch.equal(alone[n], packed[n][i:i + 1] if n in ("ht", "dh0") else packed[n][:, s:e]), (n, i)


@pytest.mark.parametrize("keep", [False, True])
def test_fp32_calls_in_a_checkpointed_segment(keep, monkeypatch):
    """Room for the intermediates of one call of three: in a checkpointed segment all three find it, since nothing is held between, and when the segment
    is run again for its backward only the first does.  The saved tensors must be the same ones both times."""
    from torch.utils.checkpoint import checkpoint
    from kda_b200 import chunk_kda, ops
    d = {n: t.cuda() for n, t in make_inputs(1, 200, 2, 64, 64, torch.float32, seed=60, backward=True).items() if t is not None}
    lv = [d[n].requires_grad_(True) for n in ("q", "k", "v", "g", "beta")]
    monkeypatch.setattr(ops, "_keep_limit", lambda index: 200 * 2 * 64 * 4 * 2 + 200 // 32 * 2 * 64 * 64 * 4)

    def segment(q, k, v, g, beta):
        for _ in range(3):
            v = chunk_kda(q, k, v, g, beta, disable_recompute=keep)[0]
        return v

    plain = torch.autograd.grad(segment(*lv), lv, d["do"])
    out = checkpoint(segment, *lv, use_reentrant=False)
    assert all(torch.equal(a, b) for a, b in zip(plain, torch.autograd.grad(out, lv, d["do"])))
    del out
    assert not ops._kept
