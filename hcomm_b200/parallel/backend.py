"""torch.distributed backend ``"hccl"``.

    import hcomm_b200.parallel.backend            # registers the backend
    torch.distributed.init_process_group("hccl", ...)

The backend object is the C++ class ``ProcessGroupHCCL`` (csrc/torch/process_group_hccl.cpp): one communicator per
process group, operators on a dedicated communication stream, ``Work.wait()`` stream-ordered.  CUDA tensors use the
GPU platform; CPU tensors are served when the library runs on its host simulator (``HCCL_SIM=1``), which is how the
backend is tested without a GPU.

The role is that of the reference's ``torch_npu`` process group over the same C API (reference: python/hccl/manage/api.py
exposes the communicator management that backend sits on).
"""
from __future__ import annotations

import torch
import torch.distributed as dist

from .._ext import extension
from ..comm import Communicator

BACKEND_NAME = "hccl"


def _create(store, rank, size, timeout):
    return extension().create_backend(store, rank, size, timeout)


def register() -> None:
    """Registers the backend with torch.distributed (idempotent)."""
    if hasattr(dist.Backend, BACKEND_NAME.upper()):
        return
    dist.Backend.register_backend(BACKEND_NAME, _create, devices=["cuda", "cpu"])


def native_backend(group=None, device: torch.device | None = None):
    """The ``ProcessGroupHCCL`` object behind a torch process group (default group when None)."""
    group = group if group is not None else dist.group.WORLD
    if device is None:
        device = torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")
    return group._get_backend(device)


def communicator_of(group=None, device: torch.device | None = None) -> Communicator:
    """The library communicator of a torch process group, for the C API and the fused operators."""
    if device is None:
        device = torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")
    return Communicator.from_handle(native_backend(group, device).comm_handle(device))


register()
