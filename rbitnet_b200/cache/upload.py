"""Small host arrays to the device without making the host wait."""
from __future__ import annotations

import numpy as np
import torch


#: up to so many bytes are copied from pageable memory (the driver takes them into a buffer of its own before the call returns)
STAGED_BYTES = 64 << 10


def upload(array: np.ndarray, device) -> torch.Tensor:
    """A tensor on ``device`` with the array's values and no part of its memory; the array may change as soon as this returns.

    On a GPU the copy is asked for in stream order and not waited for: with torch's default a copy from pageable memory ends
    with a wait for the whole stream, so that a step's second batch of rows could not be launched before its first had run.
    That the driver has read all of a small pageable source when the call returns is how it stages such copies; CUDA's documents
    say so in general terms only, and a test overwrites arrays behind a stream that is kept busy.  Larger arrays go through pinned memory (a block of torch's pool, which
    keeps it until the copy has run); small ones do not, because a block that the pool does not have yet costs more than the copy.

    Not under capture: a graph would keep the address of the array's memory and copy from it at every replay."""
    device = torch.device(device)
    t = torch.from_numpy(array)
    if device.type != "cuda":
        return t.to(device, copy=True)
    if torch.cuda.is_current_stream_capturing():
        raise RuntimeError("a host array cannot be uploaded while the stream is being captured")
    return (t if t.nbytes <= STAGED_BYTES else t.pin_memory()).to(device, non_blocking=True)


def upload_into(target: torch.Tensor, array: np.ndarray) -> None:
    """The array's values into ``target`` (contiguous, on a GPU), as ``upload`` would bring them but without a tensor between: a
    page that a sequence begins is then one small copy.  Measured at 64 sequences, one or two of which begin a page in each step: the
    tables took the host 32 us a step with a tensor between and a copy on the device after it, 19 us without."""
    if array.nbytes > STAGED_BYTES:
        target.copy_(upload(array, target.device))
        return
    if torch.cuda.is_current_stream_capturing():
        raise RuntimeError("a host array cannot be uploaded while the stream is being captured")
    target.copy_(torch.from_numpy(array), non_blocking=True)
