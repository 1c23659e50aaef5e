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
        if calls is None:
            return super().step(closure)
        for call in calls:
            hb.adam_step(*call)

    def _native_calls(self):
        if getattr(self, "grad_scale", None) is not None or getattr(self, "found_inf", None) is not None:
            return None
        calls = []
        for g in self.param_groups:
            lr, (b1, b2), eps = g["lr"], g["betas"], g["eps"]
            if (g["weight_decay"] != 0 or g["amsgrad"] or g["maximize"] or g["differentiable"]
                    or not (g["capturable"] or g["fused"])
                    or any(isinstance(v, torch.Tensor) for v in (lr, b1, b2, eps))):
                return None
            params, grads, states = [], [], []
            for p in g["params"]:
                if p.grad is None:
                    continue
                if not (p.is_cuda and p.dtype == torch.float32 and p.is_contiguous() and p.numel() > 0
                        and p.grad.dtype == torch.float32 and p.grad.layout == torch.strided
                        and (not params or p.device == params[0].device)):
                    return None
                params.append(p)
                grads.append(p.grad)
                s = self.state[p]
                if not s:
                    s["step"] = torch.zeros((), dtype=torch.float32, device=p.device)
                    s["exp_avg"] = torch.zeros_like(p)
                    s["exp_avg_sq"] = torch.zeros_like(p)
                elif not (s["step"].is_cuda and s["step"].dtype == torch.float32
                          and s["exp_avg"].is_contiguous() and s["exp_avg_sq"].is_contiguous()):
                    return None
                states.append(s)
            calls.append((params, grads, [s["exp_avg"] for s in states], [s["exp_avg_sq"] for s in states],
                          [s["step"] for s in states], lr, b1, b2, eps))
        return calls
