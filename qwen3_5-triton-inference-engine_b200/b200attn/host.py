"""Host data on its way to the device."""
from __future__ import annotations

import numpy as np
import torch


def upload(values, device, dtype=None) -> torch.Tensor:
    """A list, an array or a host tensor as a device tensor, by a copy the host does not wait for.

    A blocking copy returns when it is done, and it is done behind everything in the stream: an engine that sends lengths or slots
    that way stands still until the device is idle, and the device then until the next launches arrive.  A non-blocking one from pageable
    memory returns when the driver has the values in its own staging memory.  (Pinned memory of PyTorch's pool made every first pass 4 ms
    longer: pages are locked anew.)"""
    return torch.as_tensor(values, dtype=dtype).to(device, non_blocking=True, copy=True)


def token_array(prompts, dtype=np.int32) -> np.ndarray:
    """The tokens of all prompts behind one another."""
    from itertools import chain
    return np.fromiter(chain.from_iterable(prompts), dtype=dtype, count=sum(map(len, prompts)))
