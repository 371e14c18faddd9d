"""Performance cases of the ring-attractor operator: what a user of this framework has it compute, through its public
entry points, over the sizes it is used at.

Four kinds of call:

  train     one training step: ``dp.train_step`` on ``dp.fused_step_fn`` (forward, decode, loss, backward through time)
            followed by ``optim.FusedClipAdam.step``, the loop body of a program that trains on the fused surface
  op        the autograd operator ``ring_rnn_cuda_func`` by itself, the surface the reference's models call: forward, and
            (unless ``forward_only``) backward from the gradient of the bump history; ``input_grads`` also asks for
            dL/d(action signal) and dL/d(initial state), which is what a model with gain networks in front needs
  rollout   ``fused.ring_rnn_rollout``: decoded angles of a long sequence with nothing saved, and their angular error
  evaluate  ``evaluate.evaluate_angular_error``: the held-out evaluation, trials generated on the host included

Weights stand for a trained network: a cosine ring profile strong enough to hold a bump of activity (``GAIN``), cosine
profiles shifted by +-45 degrees for the action matrices, and a random part.  The activity then neither dies out nor
saturates over a long sequence and gradients stay well conditioned, so that two correct evaluations agree.  The global
inhibition is the reference's -0.1 up to 128 neurons and keeps that loop gain beyond (a sixteenth of that for relu, which
has no saturation to hold a bump against more).
"""
import math

import torch

from rnn_train_ring_attractor_b200 import dp, evaluate, fused, inputs, optim, ring_rnn_cuda

ACTS = ("relu", "gelu", "tanh", "silu")
GAIN = {"relu": 2.4, "gelu": 2.0, "tanh": 1.5, "silu": 2.0}
MAX_AV = 0.1 * math.pi


def _case(kind, N, B, T, activation, a_dim=2, active=2, alpha=0.1, precision="auto", ckpt_every=0, forward_only=False,
          input_grads=False, name=None):
    c = dict(kind=kind, N=N, B=B, T=T, activation=activation, a_dim=a_dim, active=active, alpha=alpha,
             precision=precision, ckpt_every=ckpt_every, forward_only=forward_only, input_grads=input_grads)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's own training script: 16 action columns of which L and R are used, batch 32: the smallest call
        _case("op", 64, 32, 40, "gelu", a_dim=16, alpha=0.15, name="op-script-n64"),
        # a training step at the reference's network size (the configuration that also runs on a CPU)
        _case("train", 120, 128, 120, "tanh", name="train-n120"),
        # a training step of the middle configuration
        _case("train", 256, 1024, 256, "relu", name="train-n256"),
        # the headline configuration: N=512, batch 4096, 512 steps
        _case("train", 512, 4096, 512, "gelu", name="train-n512"),
        # one GPU's shard of the largest network, state checkpoints every 64 steps and recompute in backward
        _case("train", 1024, 1024, 512, "tanh", ckpt_every=64, name="train-n1024-ckpt"),
        # the fp32 mode, for users who need 1e-4 parity; sizes that are multiples of nothing
        _case("train", 250, 200, 100, "silu", precision="fp32", name="train-fp32-n250"),
        # a gain-network model on the operator: gradients of the action signal and the initial state too; ragged sizes
        _case("op", 200, 1000, 150, "silu", input_grads=True, name="op-gains-n200"),
        # forward latency on two shapes of the reference's published table (every action column active)
        _case("op", 512, 256, 20, "tanh", a_dim=16, active=16, alpha=0.15, forward_only=True, name="op-table-n512-a16"),
        _case("op", 2048, 256, 20, "tanh", a_dim=16, active=16, alpha=0.15, forward_only=True, name="op-table-n2048-a16"),
        # a wide action signal at a training batch, forward and backward
        _case("op", 256, 2048, 64, "gelu", a_dim=6, active=6, name="op-wide-n256-a6"),
        # the large roll-out configuration: 65536 trials of 4000 steps, forward only
        _case("rollout", 120, 65536, 4000, "tanh", name="rollout-n120"),
        # the angular-error evaluation: 200 trials of 500 steps in batches of 50
        _case("evaluate", 120, 200, 500, "tanh", name="evaluate-n120"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same kinds and ranges; no more work than the largest listed case of its kind."""
    what = rng.choice(("train", "train", "train", "train-fp32", "op", "op", "op-gains", "table", "wide", "rollout", "evaluate"))
    act = rng.choice(ACTS)
    smooth = rng.choice(ACTS[1:])  # a random cotangent on relu's kink says little about either of two evaluations
    if what == "train":
        N = _log(rng, 48, 1024)
        B, T = _log(rng, 24, 4096), _log(rng, 24, 512)
        if N > 512:
            B = min(B, 1024)
        ckpt = rng.choice((0, 0, 0, 16, 64))
        return _case("train", N, B, T, act, ckpt_every=ckpt if ckpt < T else 0)
    if what == "train-fp32":
        return _case("train", _log(rng, 32, 256), _log(rng, 16, 256), _log(rng, 16, 100), act, precision="fp32")
    if what == "op":  # the script's surface: L and R among padding columns
        return _case("op", _log(rng, 32, 512), _log(rng, 16, 512), _log(rng, 16, 128), smooth,
                     a_dim=rng.choice((2, 4, 16)), alpha=0.15)
    if what == "op-gains":
        return _case("op", _log(rng, 48, 512), _log(rng, 32, 1024), _log(rng, 16, 150), smooth, input_grads=True)
    if what == "table":
        a = rng.choice((3, 6, 12, 16))
        return _case("op", _log(rng, 128, 2048), 256, 20, smooth, a_dim=a, active=a, alpha=0.15, forward_only=True)
    if what == "wide":
        a = rng.randint(3, 8)
        return _case("op", _log(rng, 64, 384), _log(rng, 128, 2048), _log(rng, 12, 64), smooth, a_dim=a, active=a)
    if what == "rollout":
        return _case("rollout", rng.randint(64, 128), _log(rng, 256, 65536), _log(rng, 200, 4000), rng.choice(("tanh", "gelu")))
    return _case("evaluate", rng.randint(64, 250), rng.randint(50, 200), rng.randint(100, 500), rng.choice(("tanh", "gelu")))


def _weights(c, seed):
    N, a = c["N"], c["a_dim"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    idx = torch.arange(N, dtype=torch.float32, device="cuda")
    d = 2 * math.pi * (idx[:, None] - idx[None, :]) / N
    gain, J1 = GAIN[c["activation"]], 0.1
    Wo = gain * 2 / (N * J1) * torch.cos(d) + torch.randn(N, N, generator=g, device="cuda") / math.sqrt(N)
    Wa = 0.1 * torch.randn(a, N, N, generator=g, device="cuda") / math.sqrt(N)
    for k in range(c["active"]):
        Wa[k] += gain * 2 / N * torch.cos(d + (math.pi / 4 if k % 2 == 0 else -math.pi / 4)) * 2 / c["active"]
    J0 = -0.1 * min(1.0, (16.0 if c["activation"] == "relu" else 128.0) / N)
    return Wo.contiguous(), Wa.contiguous(), J0, J1


def prepare(case, seed):
    c = dict(case)
    N, B, T, a = c["N"], c["B"], c["T"], c["a_dim"]
    Wo, Wa, J0, J1 = _weights(c, seed)
    s = dict(c=c, Wo=Wo, Wa=Wa, J0=J0, J1=J1, seed=seed)
    if c["kind"] == "evaluate":
        return s
    x = inputs.generate_on_device(B, T, N, seed=seed, max_av=MAX_AV, action_dim=a)
    A = x["A"]
    if c["active"] > 2:  # every column carries a share of the velocity, as the signal of the published table
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        A = (torch.rand(B, T, a, generator=g, device="cuda") * (A.sum(dim=2, keepdim=True) + 0.1)).contiguous()
    s.update(A=A, r_init=x["r_init"], target=x["target"])
    if c["kind"] == "train":
        s["params"] = optim.FlatRingParams(Wo, Wa, J0, J1)
        s["opt"] = optim.FusedClipAdam(s["params"].flat)
        s["buf"] = torch.empty(dp.grad_buffer_numel(N, a), dtype=torch.float32, device="cuda")
        s["step_fn"] = dp.fused_step_fn(s["params"].Wa, J0, J1, s["params"].Wo, c["alpha"], c["activation"],
                                        precision=c["precision"], ckpt_every=c["ckpt_every"])
    elif c["kind"] == "op" and not c["forward_only"]:
        g = torch.Generator(device="cuda").manual_seed(seed + 2)
        s["cot"] = torch.randn(T, B, N, generator=g, device="cuda")
        s["Wo"].requires_grad_(True)
        s["Wa"].requires_grad_(True)
        if c["input_grads"]:
            s["A"].requires_grad_(True)
            s["r_init"].requires_grad_(True)
    return s


def run(s):
    c = s["c"]
    if c["kind"] == "train":
        loss, out = dp.train_step(s["step_fn"], (s["A"], s["r_init"], s["target"]), c["N"], c["a_dim"], c["B"], c["T"],
                                  buf=s["buf"])
        norm = s["opt"].step(s["buf"][:-2])
        return {"loss": loss, "grads": s["buf"], "norm": norm, "params": s["params"].flat,
                "exp_avg": s["opt"].exp_avg, "exp_avg_sq": s["opt"].exp_avg_sq}
    if c["kind"] == "op":
        ring_rnn_cuda.set_precision(c["precision"])
        args = (s["A"], s["Wa"], s["J0"], s["J1"], s["Wo"], s["r_init"], c["alpha"], c["activation"])
        if c["forward_only"]:
            with torch.no_grad():
                return ring_rnn_cuda.ring_rnn_cuda_func(*args)
        hist = ring_rnn_cuda.ring_rnn_cuda_func(*args)
        wrt = [s["Wo"], s["Wa"]] + ([s["A"], s["r_init"]] if c["input_grads"] else [])
        return [hist.detach()] + list(torch.autograd.grad(hist, wrt, s["cot"]))
    if c["kind"] == "rollout":
        decoded, final_state = fused.ring_rnn_rollout(s["A"], s["Wa"], s["J0"], s["J1"], s["Wo"], s["r_init"], c["alpha"],
                                                      c["activation"], precision=c["precision"])
        return evaluate.angular_error(decoded, s["target"]), final_state
    return evaluate.evaluate_angular_error(s["Wa"], s["J0"], s["J1"], s["Wo"], c["alpha"], c["activation"],
                                           n_trials=c["B"], seq_len=c["T"], seed=s["seed"], precision=c["precision"])


def work(case):
    c = case
    N, B, T, a = c["N"], c["B"], c["T"], c["a_dim"]
    step = 2.0 * N * N * (1 + c["active"])  # one product of the state with every matrix in use, per sample and step
    weights = 4.0 * (1 + a) * N * N
    signal = 4.0 * B * T * a
    if c["kind"] == "train":  # inputs and target, weights and gradients, both moments and the parameters updated
        return {"bytes": signal + 4.0 * B * T + 4.0 * B * N + 8 * weights, "flops": 3 * step * B * T}
    if c["kind"] == "op":
        hist = 4.0 * T * B * N
        if c["forward_only"]:
            return {"bytes": signal + weights + 4.0 * B * N + hist, "flops": step * B * T}
        more = signal + 4.0 * B * N if c["input_grads"] else 0.0
        return {"bytes": signal + 2 * weights + 4.0 * B * N + 2 * hist + more, "flops": 3 * step * B * T}
    # roll-out and evaluation: action signal, target and initial state in, angles (their errors) out
    return {"bytes": signal + 8.0 * B * T + 8.0 * B * N + weights, "flops": step * B * T}


def tolerance(case):
    # fp32 mode: fp32 sums carried through a recurrence of some hundred steps; otherwise bf16 operands on tensor cores
    return {"rel": 1e-4} if case["precision"] == "fp32" else {"rel": 1e-2, "max": 0.5}
