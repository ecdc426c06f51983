"""Whole blocks without a graph as one native call.

A generation step's kernels take 2 to 9 us each; launched module by module from Python an operator costs 14 to 25 us and a module call a few
more.  Where nothing can tell the difference (no graph, no transform or trace, plain modules without hooks, plain bf16 parameters, one
tensor-parallel rank, no active dropout, no mask) the block's kernels are launched in the same order from C++ (``block_fwd`` and
``llama_block_fwd`` in ``csrc/bindings.cpp``, which look at the tensors); everything else runs through the modules as ever, so ``None`` is
always a safe answer.  Nothing is kept from one call for the next.
"""
import torch
from torch.nn import Parameter
from torch.nn.modules import module as _module

from libai_b200 import ops
from libai_b200.ops import functional as OF
from libai_b200.utils import distributed as dutil

_FORWARDS = {}
_CALL = torch.nn.Module.__call__


def remember(*classes):
    """The forwards that a native call stands for (a class whose ``forward`` is replaced later runs through its modules)."""
    for cls in classes:
        _FORWARDS[cls] = cls.forward


def applies(x) -> bool:
    """What holds for the call as a whole."""
    return (not torch.is_grad_enabled() and type(x) is torch.Tensor and x.dtype is torch.bfloat16 and x.dim() == 3 and ops.use_native(x)
            and OF._plain_call() and not ops.fp8_enabled() and dutil.get_dist_util().tensor_parallel_size == 1 and not _calls_are_seen())


def applies_with_graph(x) -> bool:
    """The same for a call with a graph: a block's nodes made in one call (``block_nodes``, ``llama_block_nodes`` in ``csrc/autograd_nodes.cpp``)."""
    if not (OF._graph_node(x) and x.dtype is torch.bfloat16 and x.dim() == 3 and ops.use_native(x)) or _calls_are_seen():
        return False
    topo = dutil.get_dist_util()
    return topo.tensor_parallel_size == 1 and not topo.sequence_parallel and not topo.fused_tp_comm


def _calls_are_seen() -> bool:
    """Does anything look at the call of every module: global hooks, a replaced ``Module.__call__``?"""
    return bool(_module._global_forward_hooks or _module._global_forward_pre_hooks or _module._global_backward_hooks or _module._global_backward_pre_hooks
                or torch.nn.Module.__call__ is not _CALL)


def plain(m, cls) -> bool:
    """A module of this very class whose call without a graph is its class's ``forward`` and nothing else."""
    if type(m) is not cls or cls.forward is not _FORWARDS[cls]:
        return False
    own = m.__dict__                     # (a lookup each where the attribute takes three)
    return not own["_forward_hooks"] and not own["_forward_pre_hooks"] and "_compiled_call_impl" not in own and "forward" not in own


def plain_with_graph(m, cls) -> bool:
    """The same for a call with a graph, where the module's backward hooks count too."""
    return plain(m, cls) and not m._backward_hooks and not m._backward_pre_hooks


def alone(m, cls) -> bool:
    """Would nobody notice if this module were passed by, its work joined with a neighbour's, with a graph or without?"""
    return plain_with_graph(m, cls) and not _calls_are_seen()


def parameters(*pairs):
    """``(module, name, ...)`` tuples → their parameters, or ``None`` where one is missing or of another kind (a view, a parametrization)."""
    out = []
    for m, *names in pairs:
        for name in names:
            p = m._parameters.get(name)
            if type(p) is not Parameter:
                return None
            out.append(p)
    return out


def past_pair(past, heads: int, x):
    """``(keys, values)`` of a cache that one new token may join in one kernel, ``(None, None)`` without one, else ``None``."""
    if past is None:
        return None, None
    if len(past) != 2 or x.shape[1] != 1 or not all(type(t) is torch.Tensor and t.dim() == 4 for t in past):
        return None
    b = x.shape[0]
    if b * heads < 4 and OF._cache_too_long_for_one_cluster(b * heads, past[0].shape[2], past[0].shape[3]):
        return None
    return past
