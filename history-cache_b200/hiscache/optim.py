"""Adam whose step is one kernel over all parameters (csrc/adam.cu)."""
from __future__ import annotations

import torch

import hiscache_backend as hb


class Adam(torch.optim.Adam):
    """torch.optim.Adam with the same arguments, state and state dict.

    torch's fused step gives a block 64 K values, which keeps a handful of blocks busy for the half
    million parameters of these models, and takes some 100 us on the host.  The plain case (fp32 CUDA
    parameters, device-side step counts, no weight decay, amsgrad, maximize or gradient scale) runs
    in the library; every other case runs in torch."""

    @torch.no_grad()
    def step(self, closure=None):
        calls = self._native_calls() if closure is None else None
        # several groups: all of them or none, so that torch's step never follows half of ours
        if calls is None or (len(calls) > 1 and not all(hb.adam_fits(*c[:5]) for c in calls)):
            return super().step(closure)
        for call in calls:
            if not hb.adam_step(*call):
                return super().step()

    def zero_grad(self, set_to_none=True):
        if not set_to_none:
            return super().zero_grad(False)
        for g in self.param_groups:
            for p in g["params"]:
                p.grad = None

    def _native_calls(self):
        """Arguments of hb.adam_step per parameter group, or None when torch has to do the step."""
        if getattr(self, "grad_scale", None) is not None or getattr(self, "found_inf", None) is not None:
            return None
        calls = []
        for g in self.param_groups:
            lr, (b1, b2), eps = g["lr"], g["betas"], g["eps"]
            if (g["weight_decay"] != 0 or g["amsgrad"] or g["maximize"] or g["differentiable"]
                    or not (g["capturable"] or g["fused"])
                    or any(isinstance(v, torch.Tensor) for v in (lr, b1, b2, eps))):
                return None
            params = [p for p in g["params"] if p.grad is not None]
            states = [self.state[p] for p in params]
            for p, s in zip(params, states):
                if s:
                    continue
                if not p.is_cuda or p.dtype != torch.float32:
                    return None
                s["step"] = torch.zeros((), dtype=torch.float32, device=p.device)
                s["exp_avg"] = torch.zeros_like(p)
                s["exp_avg_sq"] = torch.zeros_like(p)
            tensors = (params, [p.grad for p in params], [s["exp_avg"] for s in states],
                       [s["exp_avg_sq"] for s in states], [s["step"] for s in states])
            calls.append((*tensors, lr, b1, b2, eps))
        return calls
