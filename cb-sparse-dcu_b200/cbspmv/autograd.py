"""``torch.autograd.Function`` over the CB-SpMV C ABI (a test harness).

Y = A(vals) X where ``vals`` are the matrix's input nonzero values (the
caller's COO order) and X is (n,) or (n, k).  Backward:

* dL/dX    = A^T dL/dY, on the plan's transposed CB layout (build the plan
  with ``want_transpose=1``);
* dL/dvals = for each input nonzero k, dL/dY[row_k, :] . X[col_k, :],
  computed in input order (``adjoint_input``: the value-gradient kernel over
  the input nonzeros' rows and columns, on a second stream beside
  A^T dL/dY) -- every input is summed into exactly one stored value, so that
  value's gradient is the input's gradient.  ``adjoint`` (per stored value,
  gathered through ``input_slots``) and ``adjoint_fused`` (one launch,
  gathered through ``grad_positions_t``) compute the same.

Build the plan with ``keep_values=1`` when its initial values may all be 1:
a unit-valued plan stores no values and cannot take new ones.
"""
from __future__ import annotations

import torch


class CBSpMVFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, vals, x, plan):
        plan.set_values(vals.detach().contiguous())
        y = plan.spmv(x.detach().contiguous())
        ctx.plan = plan
        ctx.save_for_backward(x)
        return y

    @staticmethod
    def backward(ctx, gy):
        plan = ctx.plan
        (x,) = ctx.saved_tensors
        gy = gy.contiguous()
        want_gx, want_v = ctx.needs_input_grad[1], ctx.needs_input_grad[0]
        if not (want_gx or want_v):
            return None, None, None
        # both in one call: the value gradient overlaps A^T g on a second
        # stream
        gx, gvals = plan.adjoint_input(gy, x.contiguous(), want_gx=want_gx, want_gin=want_v)
        return gvals, gx, None


def cbspmv_apply(plan, vals, x):
    """Differentiable Y = A(vals) X through the plan."""
    return CBSpMVFunction.apply(vals, x, plan)
