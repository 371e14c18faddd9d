"""The persistent kernels of large batches (tiles of 128 samples) over many steps, fused loss and checkpoints included, against
the fp32 mode.  Other tests of these shapes take a handful of steps, or few samples, which run on other kernels; here every
barrier and ring slot comes round many times.

Weights hold a bump of activity (a cosine ring profile above threshold, see perf/cases.py), so that decoded angles and gradients
stay well conditioned over the sequence: 1e-2 relative, the bound of the bf16 mode."""
import math

import pytest
import torch

from oracle import ring_oracle as orc

pytestmark = pytest.mark.gpu
GAIN = {"gelu": 2.0, "tanh": 1.5, "silu": 2.0}
# batches above what small tiles and the stepwise path take
CASES = [(512, 1100, 200, "gelu", 0), (512, 1100, 200, "gelu", 64), (1024, 520, 130, "tanh", 0), (1024, 520, 130, "tanh", 32),
         (256, 4800, 100, "silu", 0), (100, 9500, 100, "tanh", 16)]


def _inputs(N, B, T, act):
    from rnn_train_ring_attractor_b200 import inputs
    g = torch.Generator().manual_seed(N)
    idx = torch.arange(N, dtype=torch.float32)
    d = 2 * math.pi * (idx[:, None] - idx[None, :]) / N
    gain, J1 = GAIN[act], 0.1
    Wo = gain * 2 / (N * J1) * torch.cos(d) + torch.randn(N, N, generator=g) / math.sqrt(N)
    Wa = 0.1 * torch.randn(2, N, N, generator=g) / math.sqrt(N)
    for k, shift in enumerate((math.pi / 4, -math.pi / 4)):
        Wa[k] += gain * 2 / N * torch.cos(d + shift)
    x = inputs.generate_on_device(B, T, N, seed=N)
    return x["A"], Wa.cuda(), -0.1 * min(1.0, 128.0 / N), J1, Wo.cuda(), x["r_init"], x["target"]


@pytest.mark.parametrize("cfg", CASES, ids=lambda c: "N%d-B%d-T%d-%s-K%d" % c)
def test_training_step_over_many_steps(cfg, achieved):
    from rnn_train_ring_attractor_b200.fused import ring_rnn_fused
    N, B, T, act, ckpt = cfg
    A, Wa, J0, J1, Wo, r0, target = _inputs(N, B, T, act)
    out = {}
    for prec in ("bf16", "fp32"):
        leaves = [t.clone().requires_grad_(True) for t in (Wo, Wa, r0)]
        loss, _, decoded, final = ring_rnn_fused(A, leaves[1], J0, J1, leaves[0], leaves[2], 0.1, act, target, precision=prec,
                                                 ckpt_every=ckpt)
        loss.backward()
        out[prec] = dict(loss=loss.detach(), decoded=decoded, final=final, dWo=leaves[0].grad, dWa=leaves[1].grad, dr0=leaves[2].grad)
    a, b = out["bf16"], out["fp32"]
    e = {k: orc.rel_err(a[k], b[k]) for k in ("loss", "final", "dWo", "dWa", "dr0")}
    e["decoded"] = float(orc.angular_error(a["decoded"].cpu(), b["decoded"].cpu()).mean())
    achieved("tiles over time N%d-B%d-T%d-%s-K%d" % cfg, **e)
    # the gradient of the initial state is what is left of delta after T products with it rounded to bf16: sqrt(T) 2^-9
    assert e.pop("dr0") < math.sqrt(T) * 2.0 ** -9
    assert all(v < 1e-2 for v in e.values()), e
