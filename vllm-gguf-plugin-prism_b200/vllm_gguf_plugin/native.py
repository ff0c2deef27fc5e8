# SPDX-License-Identifier: Apache-2.0
"""The functions that eager calls go through on their way to the kernels (csrc/eager.cpp).

They answer ``None`` for anything but plain CUDA tensors, and the caller then takes the registered
operator.  The module behind them is tied to one Python and one torch; under any other they answer
``None`` always, so every call goes through the operators, which run under every torch with the
stable ABI."""
from __future__ import annotations

import logging

try:
    from ._eager import embed, linear, linear_runs, moe, mul_mat
except ImportError as exc:
    logging.getLogger("vllm_gguf_plugin").warning("eager calls go through the operator dispatcher: %s", exc)

    def _through_the_operators(*args):
        return None

    embed = linear = linear_runs = moe = mul_mat = _through_the_operators
