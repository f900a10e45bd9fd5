"""Common plumbing of the weighted equivariant layers: optional internal weight, reshaping of
externally supplied (possibly per-sample) weights, and moving the index tables together with the
module (they are plain attributes, not buffers, exactly as in the reference:
``equitorch/nn/tensor_products.py:173-178``)."""
from __future__ import annotations

import math
from typing import Optional, Sequence

import torch
from torch import Tensor, nn
from torch.nn import Parameter

from ..tables import generate_fully_connected_tp_paths, so3_path_norms


class _WeightedTableModule(nn.Module):
    _table_attrs: Sequence[str] = ()

    def _setup_weight(self, weight_shape, internal_weights: bool, initializer) -> None:
        self.weight_shape = tuple(weight_shape)
        self.weight_numel = math.prod(self.weight_shape)
        self.internal_weights = internal_weights
        if internal_weights:
            self.weight = Parameter(torch.empty(*self.weight_shape))
            initializer(self.weight)
        else:
            self.weight = None

    def _resolve_weight(self, weight: Optional[Tensor]) -> Tensor:
        if self.internal_weights:
            assert weight is None, "Do not pass the weight when self.internal_weights is True."
            return self.weight
        assert weight is not None, "Please pass the weight when self.internal_weights is False."
        if weight.numel() > self.weight_numel:
            return weight.view(-1, *self.weight_shape)
        return weight.view(*self.weight_shape)

    def _apply(self, fn, *args, **kwargs):
        module = super()._apply(fn, *args, **kwargs)
        for name in self._table_attrs:
            setattr(module, name, getattr(self, name)._apply(fn))
        return module


class _PathModule(_WeightedTableModule):
    """A layer over paths between the irreps of two operands and an output, which kernels of their own evaluate from a plan of
    the paths (``_plan_type``) as long as the layer's tables are those of its paths."""
    _table_attrs = ("tp_info_forward", "tp_info_backward1", "tp_info_backward2")
    _plan_type = None

    def _set_paths(self, path, fan_in) -> None:
        paths = path or generate_fully_connected_tp_paths(self.irreps_out, self.irreps_in1, self.irreps_in2)
        self._paths = (list(paths), so3_path_norms(paths, self.path_norm, self.channel_norm, fan_in ** (-0.5) if fan_in else 1.0))
        self._own_tables()

    def _tables(self):
        return self.tp_info_forward, self.tp_info_backward1, self.tp_info_backward2

    def _own_tables(self, own: bool = True) -> None:
        """``own``: the layer's tables are those of its paths, in the state that they are in now."""
        scale = self.tp_info_forward.info_Mij_fwd.scale
        version = None if scale is None or scale.is_inference() else scale._version        # inference mode: none to compare
        self._path_plans, self._own = {}, ((*self._tables(), scale, version) if own else None)

    def _is_own(self) -> bool:
        if self._own is None:
            return False
        forward, backward1, backward2, scale, version = self._own
        return (self.tp_info_forward is forward and self.tp_info_backward1 is backward1 and self.tp_info_backward2 is backward2
                and (version is None or scale._version == version))

    def _path_plan(self, device):
        """The plan on ``device``, built at the first call there; ``None`` when the layer's
        own tables have been exchanged or written to, and while a stream is being captured that would have to wait for
        their copy to the device."""
        if not self._is_own():
            return None
        plan = self._path_plans.get(device)
        if plan is None and not torch.cuda.is_current_stream_capturing():
            plan = self._path_plans[device] = self._plan_type(*self._paths, self.irreps_out, self.irreps_in1, self.irreps_in2, device)
        return plan

    def _apply(self, fn, *args, **kwargs):
        own = self._is_own()
        module = super()._apply(fn, *args, **kwargs)
        module._own_tables(own)
        return module

    def __getstate__(self):
        return {**{k: v for k, v in self.__dict__.items() if k not in ("_path_plans", "_plans")}, "_own": self._is_own()}

    def __setstate__(self, state):
        super().__setstate__(state)
        self._own_tables(bool(state.get("_own", False)))          # a layer stored without its paths runs the composed products
