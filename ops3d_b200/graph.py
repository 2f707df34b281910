"""Which calls of a differentiable operator may take its C++ graph node (``csrc/autograd_nodes.h``).

The node is the fast form of the operator's ``torch.autograd.Function``: it knows reverse mode on plain tensors and nothing
else.  Whatever has to see the Function itself takes the Function.
"""
from __future__ import annotations

import torch
from torch.autograd import forward_ad


def takes_node() -> bool:
    """False under ``forward_ad.dual_level()``: the node has no forward-mode rule and would drop the tangents, where a Function
    without a ``jvp`` raises.  False under ``torch.jit.trace``: the tracer records a Function as an operation, but sees nothing
    of a node's kernels and would keep the output as a constant."""
    return forward_ad._current_level < 0 and not torch.jit.is_tracing()
