"""One training epoch of a single process as one native call (csrc/host.cpp), for the 1D, 2D and 3D models alike: on one
process their schedules all reduce to two layers on one adjacency block.

The result is what the layer functions, autograd and torch.optim.Adam produce (outputs, loss, weight gradients, updated
weights and optimizer state); what goes is their host time.  Anything outside the plain case -- several processes, timed
regions, an optimizer other than a default Adam, frozen weights, a block with a rectangular dense core -- answers None
from `plan` and takes the general path.
"""
import torch

from . import _native, ops
from .backend import CudaBackend


class _Plan:
    def __init__(self, fwd, bwd, cls_lo, cls_hi, backend):
        self.fwd, self.bwd, self.backend = fwd, bwd, backend
        self.cls_lo, self.cls_hi = cls_lo, cls_hi


def _weight_ok(w, device):
    return (isinstance(w, torch.nn.Parameter) and w.requires_grad and w.device == device and w.dtype == torch.float32
            and w.dim() == 2 and w.is_contiguous() and not w._backward_hooks)


def _adam_state(optimizer, w1, w2):
    """States (exp_avg, exp_avg_sq, step) of both weights and the options of a default torch.optim.Adam over [w1, w2], created
    as its first step would create them; None for any other optimizer."""
    if type(optimizer) is not torch.optim.Adam or len(optimizer.param_groups) != 1:
        return None
    g = optimizer.param_groups[0]
    if len(g["params"]) != 2 or g["params"][0] is not w1 or g["params"][1] is not w2:
        return None
    if g["weight_decay"] != 0 or g["amsgrad"] or g["maximize"] or g["capturable"] or g["differentiable"] or g["fused"] or \
            isinstance(g["lr"], torch.Tensor) or isinstance(g["betas"][0], torch.Tensor) or \
            optimizer._optimizer_step_pre_hooks or optimizer._optimizer_step_post_hooks:
        return None
    states = []
    for w in (w1, w2):
        s = optimizer.state[w]
        if not s:
            s["step"] = torch.tensor(0.0, dtype=torch.float32)
            s["exp_avg"] = torch.zeros_like(w, memory_format=torch.preserve_format)
            s["exp_avg_sq"] = torch.zeros_like(w, memory_format=torch.preserve_format)
        if not (s["exp_avg"].is_contiguous() and s["exp_avg_sq"].is_contiguous()) or s["step"].is_cuda or \
                s["step"].dtype != torch.float32:
            return None
        states.append(s)
    if float(states[0]["step"]) != float(states[1]["step"]):
        return None
    return states, g


def plan(backend, fwd, bwd, cls_lo, cls_hi):
    """The constant part of a model's epochs, or None where the general path has to run."""
    if type(backend) is not CudaBackend:
        return None
    for b in (fwd, bwd):
        if not isinstance(b, ops.CsrBlock) or b.n != b.m or (b.tiles is None and b._rect[0] is not None):
            return None
    return _Plan(fwd, bwd, int(cls_lo), int(cls_hi), backend)


def train(p, model, x, y, mask, count, min_width=False):
    """Run one epoch of `model` (weights, optimizer, last_loss) on features x, labels y and train mask by plan p, the loss a
    mean over `count` rows, sparse products at the narrower width of a layer if `min_width`; the outputs, or None to decline."""
    w1, w2 = model.weight1, model.weight2
    if count <= 0 or not (_weight_ok(w1, x.device) and _weight_ok(w2, x.device)):
        return None
    state = _adam_state(model.optimizer, w1, w2)
    host = _native.host()
    adam, hook = None, None
    if state is not None:
        (s1, s2), g = state
        adam = host.Adam(s1["exp_avg"], s1["exp_avg_sq"], s1["step"], s2["exp_avg"], s2["exp_avg_sq"], s2["step"], g["lr"],
                         g["betas"][0], g["betas"][1], g["eps"])
    if p.backend.spmm_events is not None:
        hook = _event_hook(p)
    out, loss, g1, g2, launches = host.epoch(p.fwd.address(), p.bwd.address(), x, w1.detach(), w2.detach(), y.contiguous(),
                                             mask.contiguous(), count, p.cls_lo, p.cls_hi, bool(model.rt.activations), min_width, adam, hook)
    ops.LAUNCHES[0] += launches
    w1.grad, w2.grad = g1, g2
    if state is not None:
        model.optimizer._opt_called = True        # what lr schedulers look at
        torch.autograd.graph.increment_version((w1, w2))
    else:
        model.optimizer.step()
    model.last_loss = loss
    return out


def _event_hook(p):
    """Brackets every sparse product with CUDA events, as CudaBackend.spmm does while it is being timed."""
    start = []

    def hook(begin, backward, width):
        event = torch.cuda.Event(enable_timing=True)
        event.record()
        if begin:
            start.append(event)
        else:
            p.backend.spmm_events.append((p.bwd if backward else p.fwd, width, 0.0, start.pop(), event))
    return hook
