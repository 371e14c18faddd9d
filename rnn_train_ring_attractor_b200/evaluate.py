"""Angular-error evaluation of a ring-attractor parameter set on held-out synthetic trials, on the fused forward.

Follows the evaluation block of compare/compare_models_fair.py:120-175: 200 test sequences of 500 steps in batches of
50, initial Gaussian bump at the first target angle, decoded angle from the population vector, circular error, and the
four statistics the script prints (mean, std, max, mean error at the final step).
"""
import math

import torch
from torch.autograd import forward_ad

from . import _lib
from .fused import ring_rnn_rollout
from .inputs import trials_from_host_draws
from .ring_rnn_cuda import on_device, stream_of


def _plain(t):
    """An ordinary contiguous fp32 CUDA tensor that nothing differentiates, batches or traces."""
    return (type(t) is torch.Tensor and t.is_cuda and t.dtype == torch.float32 and t.is_contiguous()
            and not (t.requires_grad and torch.is_grad_enabled()) and not torch._C._functorch.is_functorch_wrapped_tensor(t))


def angular_error(pred, target):
    """Circular |pred - target| in [0, pi] (compare/compare_models_fair.py:15-20)."""
    # one kernel instead of five passes over the tensors: 65536 x 4000 angles in 0.5 instead of 2 ms
    if (_plain(pred) and _plain(target) and pred.device == target.device and pred.shape == target.shape and pred.numel() > 0
            and forward_ad._current_level < 0 and torch._C._len_torch_dispatch_stack() == 0 and not torch.compiler.is_compiling()
            and not torch.jit.is_tracing()):
        out = torch.empty_like(pred)
        with on_device(pred.device):
            _lib.check(_lib.lib().ringrnn_angular_error(pred.numel(), pred.data_ptr(), target.data_ptr(), out.data_ptr(),
                                                        stream_of(pred.device)))
        return out
    d = torch.abs(pred - target) % (2 * math.pi)
    return torch.minimum(d, 2 * math.pi - d)


TRIAL_STEPS = 1 << 22  # trials x steps in hand at a time: what the roll-out of one stretch holds is about 28 bytes per step


def evaluate_angular_error(Wa, J0, J1, Wo, alpha, activation, n_trials=200, seq_len=500, batch=50, seed=123,
                           max_av=0.1 * math.pi, precision=None):
    """dict(mean, std, max, final_mean, errors[n_trials, seq_len]) in radians for the given weights (device tensors).
    ``batch`` trials are drawn at a time (it decides which trials a seed stands for); whole batches are rolled out together,
    as many as ``TRIAL_STEPS`` allows and at least one."""
    g = torch.Generator().manual_seed(seed)
    per = max(1, TRIAL_STEPS // max(1, batch * seq_len)) * batch
    errs = []
    for lo in range(0, n_trials, per):
        x = trials_from_host_draws(min(per, n_trials - lo), seq_len, Wo.shape[0], batch, max_av, g, Wo.device)
        decoded, _ = ring_rnn_rollout(x["A"], Wa, J0, J1, Wo, x["r_init"], alpha, activation, precision=precision)
        errs.append(angular_error(decoded, x["target"]))
    e = errs[0] if len(errs) == 1 else torch.cat(errs, dim=0)
    mean, std, top, final = torch.stack((e.mean(), e.std(), e.max(), e[:, -1].mean())).tolist()
    return {"mean": mean, "std": std, "max": top, "final_mean": final, "errors": e}
