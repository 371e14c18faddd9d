"""Edges of the kernels whose CTAs own few samples, and of the host-side compositions, on the GPU.

Tolerances: bf16 mode 1e-2 and fp32 mode 1e-4 relative, the bounds of the parity tests (two bf16 roundings of 2^-9 per
product, fp32 sums over at most a few thousand terms); what two entry points compute with the same kernels must be equal."""
import math
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from oracle import ring_oracle as orc  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = {"fp32": 1e-4, "bf16": 1e-2}


def _case(N, B, T, a_dim, seed):
    g = torch.Generator().manual_seed(seed)
    s = 1.0 / math.sqrt(N)
    return (torch.rand(B, T, a_dim, generator=g), torch.randn(a_dim, N, N, generator=g) * s,
            torch.randn(N, N, generator=g) * s, torch.rand(B, N, generator=g) - 0.5, torch.randn(T, B, N, generator=g))


# neurons around the 128-lane and two-CTA limits; batches around 16, 32, 64 samples per unit (148 or 74 units resident), the
# largest that train on them, and beyond; steps around the eight whose scalars are staged at a time; J1 = 0 (no ratio to J1)
LANE = [(1, 1, 1, 2, "tanh", -0.1, 0.1), (2, 17, 8, 1, "silu", -0.1, 0.1), (127, 16, 9, 2, "gelu", -0.1, 0.1),
        (128, 2369, 7, 2, "tanh", -0.07, 0.3), (129, 15, 16, 2, "silu", -0.1, 0.1), (255, 1185, 3, 2, "gelu", -0.031, 0.1),
        (256, 2400, 9, 2, "tanh", -0.05, 0.0), (120, 9500, 2, 2, "silu", 0.0, 0.1), (100, 20001, 3, 2, "tanh", -0.1, 0.1),
        (90, 9472, 3, 2, "gelu", -0.1, 0.1), (192, 4736, 2, 2, "silu", -0.05, 0.1),
        # four CTAs: neurons around 256 and 512, one and several rounds of 33 clusters of 16 samples, the last batch taken
        (257, 1, 1, 2, "tanh", -0.1, 0.1), (384, 17, 9, 1, "silu", -0.05, 0.1), (510, 33, 8, 2, "gelu", -0.013, 0.1),
        (512, 1056, 3, 2, "tanh", -0.02, 0.1), (300, 1057, 2, 2, "tanh", -0.02, 0.1), (480, 528, 2, 2, "silu", -0.02, 0.1)]
# fp32 clusters: one CTA, two, four, eight; a last CTA with few neurons; several column counts; no shape that fits
CLUSTER = [(16, 3, 2, 2, "tanh", -0.1, 0.1), (33, 40, 5, 3, "silu", -0.1, 0.1), (97, 9, 4, 2, "gelu", -0.1, 0.1),
           (200, 300, 3, 2, "tanh", -0.1, 0.1), (257, 70, 3, 1, "silu", -0.05, 0.2), (320, 33, 2, 2, "tanh", -0.04, 0.1),
           (250, 40, 3, 2, "gelu", -0.05, 0.1),
           # more tiles than resident clusters (148 of one CTA, 74 of two, 33 of four, 15 of eight): a cluster runs several
           (16, 5000, 2, 2, "tanh", -0.1, 0.1), (160, 1300, 2, 2, "silu", -0.05, 0.1), (200, 1000, 3, 2, "gelu", -0.05, 0.1),
           (250, 600, 3, 2, "silu", -0.05, 0.1),
           # a forward on clusters and a reverse pass on single CTAs, both on single CTAs
           (200, 3000, 2, 2, "tanh", -0.05, 0.1), (200, 4000, 2, 2, "silu", -0.05, 0.1)]


# one GEMM per step (more than two action columns): neurons off and on multiples of four (single and 16-byte accesses) and
# beyond one round of 512 threads x 4 neurons, one and several K splits, and a batch that takes the concatenated operand
STEPWISE = [(65, 3, 2, 3, "tanh", -0.1, 0.1), (130, 129, 3, 4, "silu", -0.1, 0.1), (384, 200, 3, 8, "gelu", -0.05, 0.1),
            (600, 1900, 2, 3, "tanh", -0.02, 0.1), (2180, 5, 2, 3, "tanh", -0.01, 0.1), (513, 512, 2, 2, "tanh", -0.02, 0.1),
            (250, 2048, 2, 6, "tanh", -0.05, 0.1), (500, 1152, 2, 4, "silu", -0.02, 0.1)]

# persistent tiles of 128 samples with several weight groups, with two K rounds, and beyond the batches of the small tiles: the
# smallest batches that train on them
GENERIC = [(256, 2060, 3, 5, "silu", -0.05, 0.1), (500, 2049, 2, 7, "gelu", -0.02, 0.1), (1000, 513, 3, 2, "tanh", -0.02, 0.1),
           (100, 1025, 3, 9, "tanh", -0.1, 0.1), (200, 1025, 2, 5, "gelu", -0.05, 0.1), (500, 1153, 2, 3, "silu", -0.02, 0.1),
           (128, 9473, 3, 2, "gelu", -0.07, 0.1), (256, 4737, 3, 2, "tanh", -0.05, 0.1), (512, 1057, 4, 2, "gelu", -0.02, 0.1),
           (480, 529, 3, 2, "tanh", -0.02, 0.1), (800, 385, 2, 2, "silu", -0.02, 0.1), (512, 1200, 3, 16, "gelu", -0.02, 0.1)]


@pytest.mark.parametrize("prec,shape", [("bf16", s) for s in LANE + STEPWISE + GENERIC] + [("fp32", s) for s in CLUSTER],
                         ids=lambda v: v if isinstance(v, str) else "N%d-B%d-T%d-a%d-%s" % v[:5])
def test_small_tile_kernels_match_the_oracle(prec, shape):
    from gpu_helpers import canaries_intact, run_backward, run_forward
    N, B, T, a_dim, act, J0, J1 = shape
    A, Wa, Wo, r0, cot = _case(N, B, T, a_dim, N + B)
    f64 = [x.double() for x in (A, Wa, Wo, r0, cot)]
    hist = orc.ring_forward_lean(f64[0], f64[1], J0, J1, f64[2], f64[3], 0.1, act)
    ref = orc.ring_backward_manual(f64[4], f64[0], f64[1], J0, J1, f64[2], hist, f64[3], 0.1, act)
    dev = [x.cuda() for x in (A, Wa, Wo, r0)]
    f = run_forward(*dev, J0, J1, 0.1, act, prec, None, history=True, decode=True)
    b = run_backward(*dev, J0, J1, 0.1, act, f, grad_output=cot.cuda(), prec=prec)
    assert all(canaries_intact(x) for x in f["backs"] + b["backs"])
    tol = TOL[prec]
    assert orc.rel_err(f["hist"], hist) < tol
    for k, name in (("dWo", "dWo"), ("dWa", "dWa"), ("dr_init", "dr_init"), ("dA", "dA")):
        assert orc.rel_err(b[k], ref[name]) < tol, k
    u, v = f["u"].cpu().double(), f["v"].cpu().double()
    h = f["hist"].cpu().double()  # the decode sums belong to this history: fp32 sums over N terms
    for k, want in (("x", h @ u), ("y", h @ v), ("ta", h.abs().sum(2))):
        scale = (h.abs() @ (u.abs() if k == "x" else v.abs() if k == "y" else torch.ones(N, dtype=torch.float64))).T
        assert float(((f[k].cpu().double() - want.T).abs() / scale.clamp(min=1e-30)).max()) < (N + 8) * 2.0 ** -24, k


# forward calls that save nothing may run on other kernels than those that do: both sides of each line
INFER = [(100, 20001, 3, 2, "tanh"), (64, 9473, 9, 2, "gelu"), (256, 4736, 3, 2, "silu"), (256, 4737, 4, 2, "gelu"),
         (400, 529, 3, 2, "tanh"), (400, 1056, 2, 2, "gelu"), (400, 1057, 2, 2, "gelu"), (1000, 384, 3, 2, "tanh"), (1000, 385, 3, 2, "tanh"), (1000, 512, 3, 2, "silu"), (64, 33, 5, 3, "silu"), (128, 1, 3, 16, "gelu"),
         (128, 1025, 3, 16, "gelu"), (256, 1024, 3, 6, "tanh"), (256, 2048, 3, 6, "tanh"), (500, 1152, 3, 4, "silu"),
         (500, 1153, 3, 4, "silu"), (300, 1025, 2, 5, "tanh")]


@pytest.mark.parametrize("shape", INFER, ids=lambda v: "N%d-B%d-T%d-a%d-%s" % v)
def test_forward_that_saves_nothing(shape):
    from gpu_helpers import canaries_intact, run_forward
    N, B, T, a_dim, act = shape
    J0, J1 = -0.1 * min(1.0, 64.0 / N), 0.1
    A, Wa, Wo, r0, _ = _case(N, B, T, a_dim, N + B)
    rows = sorted({0, 1, B // 2, B - 1} & set(range(B)))  # samples do not interact
    f64 = [x.double() for x in (A[rows], Wa, Wo, r0[rows])]
    want = orc.ring_forward_lean(f64[0], f64[1], J0, J1, f64[2], f64[3], 0.1, act)
    dev = [x.cuda() for x in (A, Wa, Wo, r0)]
    for history in (False, True):
        f = run_forward(*dev, J0, J1, 0.1, act, "bf16", None, history=history, decode=True, save=False)
        assert all(canaries_intact(x) for x in f["backs"])
        if history:
            assert orc.rel_err(f["hist"][:, rows], want) < TOL["bf16"]
        assert orc.rel_err(f["final"][rows], want[-1]) < TOL["bf16"]
        u, v = f["u"].cpu().double(), f["v"].cpu().double()
        for k, w in (("x", u), ("y", v)):
            scale = (want.abs() @ w.abs()).T
            assert float(((f[k][rows].cpu().double() - (want @ w).T).abs() / scale).max()) < 3 * TOL["bf16"], k
        assert orc.rel_err(f["ta"][rows], want.abs().sum(2).T) < TOL["bf16"]


@pytest.mark.parametrize("N,B,T", [(250, 600, 3), (32, 2100, 1000)])
def test_fp32_backward_from_the_librarys_own_history(N, B, T):
    """Without a history of the caller's the forward keeps one, and F'(re) of every step beside it up to 256 MB; otherwise the
    reverse pass forms F' from the history.  The same arithmetic either way: the same bits."""
    from gpu_helpers import canaries_intact, run_backward, run_forward
    A, Wa, Wo, r0, cot = (t.cuda() for t in _case(N, B, T, 2, 7))
    out = []
    for history in (True, False):
        f = run_forward(A, Wa * 0.3, Wo, r0, -0.03, 0.1, 0.1, "tanh", "fp32", history=history)
        out.append(run_backward(A, Wa * 0.3, Wo, r0, -0.03, 0.1, 0.1, "tanh", f, grad_output=cot))
        assert all(canaries_intact(x) for x in f["backs"] + out[-1]["backs"])
    for k in ("dWo", "dWa", "dJ", "dr_init", "dA"):
        assert torch.isfinite(out[0][k]).all() and torch.equal(out[0][k], out[1][k]), k


def test_more_steps_than_a_grid_has_rows():
    """65535 is the largest extent of a grid's second dimension: sequences beyond it on the one-GEMM-per-step path, against
    the fp32 mode.  Bound: weights, state and delta are rounded to bf16 (2^-9 each), and what a step gets wrong the next ones
    amplify by 1 / (1 - g), g the gain of the step's matrix: about 0.3 with the action matrices at a quarter of their size
    (three of spectral radius 1/4, signal 1/2 on average).  3 * 2^-9 / 0.7 = 8e-3 < 1e-2."""
    from rnn_train_ring_attractor_b200 import ring_rnn_cuda as op
    N, B, T = 16, 2, 65538
    A, Wa, Wo, r0, cot = (t.cuda() for t in _case(N, B, T, 3, 3))
    Wa *= 0.25
    Wo.requires_grad_(True), Wa.requires_grad_(True)
    got = {}
    for prec in ("bf16", "fp32"):
        op.set_precision(prec)
        try:
            hist = op.ring_rnn_cuda_func(A, Wa, -0.1, 0.1, Wo, r0, 0.1, "tanh")
            got[prec] = [hist.detach()] + list(torch.autograd.grad(hist, [Wo, Wa], cot))
        finally:
            op.set_precision("auto")
    for a, b in zip(got["bf16"], got["fp32"]):
        assert orc.rel_err(a, b) < TOL["bf16"]
    assert orc.rel_err(got["bf16"][0][-3:], got["fp32"][0][-3:]) < TOL["bf16"]


def test_several_waves_of_ctas_per_step_back_to_back():
    """One GEMM per step of 544 CTAs and row kernels of 1024 blocks, forward and reverse, calls following one another without a
    pause: the kernels' order is the stream's alone.  Sums in fixed order: every call gives the same bits."""
    from rnn_train_ring_attractor_b200 import ring_rnn_cuda as op
    N, B, T, a_dim = 2048, 1000, 20, 16
    g = torch.Generator(device="cuda").manual_seed(0)
    s = 0.5 / math.sqrt(N)
    A, r0 = torch.rand(B, T, a_dim, generator=g, device="cuda"), torch.rand(B, N, generator=g, device="cuda") - 0.5
    Wa = (torch.randn(a_dim, N, N, generator=g, device="cuda") * (s / 8)).requires_grad_(True)
    Wo = (torch.randn(N, N, generator=g, device="cuda") * s).requires_grad_(True)
    cot = torch.randn(T, B, N, generator=g, device="cuda")
    first = None
    for _ in range(6):
        hist = op.ring_rnn_cuda_func(A, Wa, -0.003, 0.1, Wo, r0, 0.1, "silu")
        out = [hist.detach()] + list(torch.autograd.grad(hist, [Wo, Wa], cot))
        first = first or out
    assert all(torch.isfinite(x).all() and torch.equal(x, y) for x, y in zip(first, out))


@pytest.mark.parametrize("a_dim,cols", [(3, [0, 2]), (16, [0, 1]), (16, []), (64, [5, 63]), (7, list(range(7)))])
def test_active_columns(a_dim, cols):
    from rnn_train_ring_attractor_b200.ring_rnn_cuda import active_columns
    A = torch.zeros(37, 61, a_dim, device="cuda")
    for k in cols:
        A[(k * 5) % 37, (k * 7) % 61, k] = -1e-30
    assert active_columns(A) == cols


@pytest.mark.parametrize("n,batch,T", [(200, 50, 500), (7, 3, 11), (5, 4, 2)])
def test_trials_from_host_draws_are_the_host_generators(n, batch, T):
    from rnn_train_ring_attractor_b200 import inputs
    x = inputs.trials_from_host_draws(n, T, 120, batch, 0.1 * math.pi, torch.Generator().manual_seed(4), "cuda")
    g = torch.Generator().manual_seed(4)
    parts = [inputs.generate_av(batch, T, generator=g) for _ in range((n + batch - 1) // batch)]
    av, angle = (torch.cat(p)[:n] for p in zip(*parts))
    assert torch.equal(x["A"].cpu(), inputs.av_to_action_signal(av, 0.1 * math.pi))
    d = (x["target"].cpu() - angle).abs()
    assert float(torch.minimum(d, 2 * math.pi - d).max()) < 4e-6  # a few ulp of 2 pi
    assert orc.rel_err(x["r_init"], inputs.initial_bump_gaussian(angle[:, 0], 120)) < 1e-5


def test_equal_ordering_draws_rank_as_on_the_host():
    """24-bit draws: of 1800 per trial, one trial in ten has two that are equal, and which of them comes first decides whether
    a step moves.  Bit for bit the host generator's signal."""
    from rnn_train_ring_attractor_b200 import inputs
    n, batch, T = 203, 7, 2000
    x = inputs.trials_from_host_draws(n, T, 16, batch, 0.3, torch.Generator().manual_seed(1), "cuda")
    g = torch.Generator().manual_seed(1)
    av, angle = (torch.cat(p)[:n] for p in zip(*[inputs.generate_av(batch, T, max_av=0.3, generator=g) for _ in range(29)]))
    assert torch.equal(x["A"].cpu(), inputs.av_to_action_signal(av, 0.3))
    d = (x["target"].cpu() - angle).abs()
    assert float(torch.minimum(d, 2 * math.pi - d).max()) < 2e-5  # a few ulp of sums up to 32


@pytest.mark.parametrize("T,ratio,max_av", [(40, 0.1, -0.3), (60000, 0.9, 0.1), (12000, 0.1, 0.1)])
def test_trials_the_device_does_not_rank_come_from_the_host(T, ratio, max_av):
    """A negative max_av, a trial whose velocities and ordering draws together exceed shared memory, more than 8192 draws."""
    from rnn_train_ring_attractor_b200 import inputs
    x = inputs.trials_from_host_draws(3, T, 24, 2, max_av, torch.Generator().manual_seed(4), "cuda", ratio)
    g = torch.Generator().manual_seed(4)
    av, angle = (torch.cat(p)[:3] for p in zip(*[inputs.generate_av(2, T, ratio, max_av=max_av, generator=g) for _ in range(2)]))
    assert torch.equal(x["A"].cpu(), inputs.av_to_action_signal(av, max_av)) and torch.equal(x["target"].cpu(), angle)


def test_evaluation_rolls_out_whole_batches_up_to_a_bound(monkeypatch):
    """The trials in hand at a time are bounded, and how many they are changes nothing."""
    from rnn_train_ring_attractor_b200 import evaluate, inputs
    Wo, Wl, Wr = (w.cuda() for w in inputs.ideal_weights(24))
    sizes = []
    inner = evaluate.ring_rnn_rollout

    def rollout(A, *args, **kw):
        sizes.append(A.shape[0] * A.shape[1])
        return inner(A, *args, **kw)

    monkeypatch.setattr(evaluate, "ring_rnn_rollout", rollout)
    args = (torch.stack([Wl, Wr]), -0.1, 0.1, Wo, 0.1, "tanh")
    evaluate.evaluate_angular_error(*args, n_trials=9000, seq_len=1000, batch=50)
    assert max(sizes) <= 1 << 22 and sum(sizes) == 9000 * 1000
    del sizes[:]
    once = evaluate.evaluate_angular_error(*args, n_trials=23, seq_len=30, batch=4)
    assert sizes == [23 * 30]
    monkeypatch.setattr(evaluate, "TRIAL_STEPS", 300)
    parts = evaluate.evaluate_angular_error(*args, n_trials=23, seq_len=30, batch=4)
    assert sizes[1:] == [8 * 30, 8 * 30, 7 * 30]
    assert torch.equal(once["errors"], parts["errors"])


def test_rollout_result_keeps_nothing_else_alive():
    from rnn_train_ring_attractor_b200.fused import ring_rnn_rollout
    case = orc.make_case(24, 6, 5, "tanh", seed=2)
    A, Wa, Wo, r0 = (t.cuda() for t in (case.A, case.Wa, case.Wo, case.r_init))
    decoded, _ = ring_rnn_rollout(A, Wa, -0.1, 0.1, Wo, r0, 0.1, "tanh")
    assert decoded.shape == (6, 5) and decoded.untyped_storage().nbytes() == 4 * decoded.numel()


@pytest.mark.parametrize("n", [1, 5, 4096, 100003])
def test_angles_and_errors(n):
    from rnn_train_ring_attractor_b200 import _lib
    from rnn_train_ring_attractor_b200.evaluate import angular_error
    g = torch.Generator().manual_seed(n)
    x, y = torch.randn(n, generator=g).cuda(), torch.randn(n, generator=g).cuda()
    out = torch.empty(n, device="cuda")
    _lib.check(_lib.lib().ringrnn_decode_angles(n, x.data_ptr(), y.data_ptr(), out.data_ptr(), None))
    want = torch.remainder(torch.atan2(y.double(), x.double()), 2 * math.pi)
    d = (out.double() - want).abs()
    assert float(torch.minimum(d, 2 * math.pi - d).max()) < 2e-6 and float(out.min()) >= 0 and float(out.max()) < 2 * math.pi
    same = x.clone()
    _lib.check(_lib.lib().ringrnn_decode_angles(n, same.data_ptr(), y.data_ptr(), same.data_ptr(), None))
    assert torch.equal(same, out)
    t = (torch.rand(n, generator=g) * 20 - 10).cuda()
    e = (out.double() - t.double()).abs() % (2 * math.pi)
    assert float((angular_error(out, t).double() - torch.minimum(e, 2 * math.pi - e)).abs().max()) < 4e-6


@pytest.mark.parametrize("N,B,T,prec,ckpt", [(40, 20, 12, None, 0), (200, 33, 9, None, 4), (300, 130, 5, None, 0), (60, 9, 7, "fp32", 0)])
def test_one_call_training_step_equals_the_autograd_surface(N, B, T, prec, ckpt):
    from rnn_train_ring_attractor_b200 import dp
    from rnn_train_ring_attractor_b200.fused import ring_rnn_fused
    case = orc.make_case(N, B, T, "tanh", seed=2)
    A, Wa, Wo, r0, tgt = (t.cuda() for t in (case.A, case.Wa, case.Wo, case.r_init, case.target))
    buf = torch.full((dp.grad_buffer_numel(N, 2),), float("nan"), device="cuda")
    loss, out = dp.train_step(dp.fused_step_fn(Wa, -0.1, 0.1, Wo, 0.1, "tanh", precision=prec, ckpt_every=ckpt), (A, r0, tgt), N,
                              2, B, T, buf=buf)
    want = torch.empty_like(buf)
    Wa.requires_grad_(True), Wo.requires_grad_(True)
    l2, parts, _, _ = ring_rnn_fused(A, Wa, -0.1, 0.1, Wo, r0, 0.1, "tanh", tgt, precision=prec, grad_buffer=want,
                                     ckpt_every=ckpt)
    l2.backward()
    assert torch.equal(buf[:-2], want[:-2]) and torch.equal(buf[-2:], parts)
    assert abs(float(loss) - float(l2)) <= 2.0 ** -22 * abs(float(l2))


@pytest.mark.parametrize("N,T", [(64, 8), (200, 12)])
@pytest.mark.parametrize("prec", ["fp32", "bf16"])
def test_weights_may_start_at_any_float(N, T, prec):
    from rnn_train_ring_attractor_b200.fused import ring_rnn_fused
    case = orc.make_case(N, 20, T, "tanh", seed=4)
    A, Wa, Wo, r0, tgt = (t.cuda() for t in (case.A, case.Wa, case.Wo, case.r_init, case.target))

    def shifted(t):
        room = torch.empty(t.numel() + 1, device="cuda")
        return room[1:].view(t.shape).copy_(t)

    def grads(Wa, Wo):
        Wa, Wo = Wa.detach().requires_grad_(True), Wo.detach().requires_grad_(True)
        loss, _, decoded, _ = ring_rnn_fused(A, Wa, -0.1, 0.1, Wo, r0, 0.1, "tanh", tgt, precision=prec)
        loss.backward()
        return loss.detach(), decoded, Wa.grad, Wo.grad

    for a, b in zip(grads(Wa, Wo), grads(shifted(Wa), shifted(Wo))):
        assert torch.equal(a, b)


def test_step_function_called_directly():
    """Loss parts are the caller's to keep, the buffer may be left out, and weights are looked up at each call."""
    from rnn_train_ring_attractor_b200 import dp
    case = orc.make_case(40, 20, 6, "tanh", seed=5)
    A, Wa, Wo, r0, tgt = (t.cuda() for t in (case.A, case.Wa, case.Wo, case.r_init, case.target))
    Wo = torch.nn.Parameter(Wo)
    step = dp.fused_step_fn(Wa, -0.1, 0.1, Wo, 0.1, "tanh")
    buf = torch.zeros(dp.grad_buffer_numel(40, 2), device="cuda")
    first = step((A, r0, tgt), 1.0 / 120, buf)
    kept = first.clone()
    buf.zero_()
    assert torch.equal(first, kept) and torch.equal(step((A, r0, tgt), 1.0 / 120, None), kept)
    Wo.data = Wo.data * 3.0
    changed = step((A, r0, tgt), 1.0 / 120, buf)
    assert torch.equal(dp.fused_step_fn(Wa, -0.1, 0.1, Wo.detach(), 0.1, "tanh")((A, r0, tgt), 1.0 / 120, buf), changed)
    assert not torch.equal(changed, kept)


@pytest.mark.parametrize("through_train_step", [False, True])
def test_step_function_reaches_what_requires_grad(through_train_step):
    """A signal out of a gain network, a learnt initial state and trained J0 / J1 receive their gradients."""
    from rnn_train_ring_attractor_b200 import dp
    from rnn_train_ring_attractor_b200.fused import ring_rnn_fused
    N, B, T = 40, 20, 6
    case = orc.make_case(N, B, T, "tanh", seed=6)
    A0, Wa, Wo, r0, tgt = (t.cuda() for t in (case.A, case.Wa, case.Wo, case.r_init, case.target))

    def leaves():
        return [torch.ones(2, device="cuda", requires_grad=True), r0.clone().requires_grad_(True)] + [
            torch.tensor(x, device="cuda", requires_grad=True) for x in (-0.1, 0.1)]

    gain, r, J0, J1 = got = leaves()
    buf = torch.full((dp.grad_buffer_numel(N, 2),), float("nan"), device="cuda")
    step = dp.fused_step_fn(Wa, J0, J1, Wo, 0.1, "tanh")
    if through_train_step:
        dp.train_step(step, (A0 * gain, r, tgt), N, 2, B, T, buf=buf)
        parts = buf[-2:]
    else:
        parts = step((A0 * gain, r, tgt), 1.0 / (B * T), buf)
    gain, r, J0, J1 = want = leaves()
    ref = torch.empty_like(buf)
    loss, ref_parts, _, _ = ring_rnn_fused(A0 * gain, Wa.requires_grad_(True), J0, J1, Wo.requires_grad_(True), r, 0.1, "tanh", tgt,
                                           grad_buffer=ref)
    loss.backward()
    assert torch.equal(buf[:-2], ref[:-2]) and torch.equal(parts, ref_parts)
    for a, b in zip(got, want):
        assert a.grad is not None and torch.equal(a.grad, b.grad)


def test_angular_error_transforms():
    from torch.autograd import forward_ad
    from rnn_train_ring_attractor_b200.evaluate import angular_error
    p, t = torch.tensor([0.5, 3.0], device="cuda"), torch.tensor([[0.25, 6.0], [1.0, 1.0]], device="cuda")
    want = torch.stack([angular_error(p, row) for row in t])
    assert torch.allclose(torch.vmap(angular_error, in_dims=(None, 0))(p, t), want, atol=4e-6)
    with forward_ad.dual_level():
        out = forward_ad.unpack_dual(angular_error(forward_ad.make_dual(p, torch.ones_like(p)), t[0]))
        assert out.tangent is not None and torch.equal(out.tangent.cpu(), torch.tensor([1.0, -1.0]))
    assert torch.equal(torch.func.grad(lambda x: angular_error(x, t[0]).sum())(p).cpu(), torch.tensor([1.0, -1.0]))
