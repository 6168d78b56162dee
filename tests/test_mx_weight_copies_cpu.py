"""Block-scaled copies of expert weights belong to a tensor, not to the address that it has."""
import numpy as np
import torch

from pisceslx_b200.ops import moe as moe_ops
from pisceslx_b200.quant import fp8


def test_a_tensor_at_a_reused_address_gets_its_own_copy(monkeypatch):
    made = []
    monkeypatch.setattr(fp8, "quantize_mx", lambda x: made.append(1) or (x.clone(), x.clone()))
    memory = np.ones((2, 4, 8), dtype=np.float32)
    first = torch.from_numpy(memory)
    assert moe_ops._mx_weight(first)[0] is moe_ops._mx_weight(first)[0] and len(made) == 1
    first.add_(1)
    assert torch.equal(moe_ops._mx_weight(first)[0], first) and len(made) == 2
    kept, address = len(moe_ops._MX_WEIGHTS), first.data_ptr()
    second = torch.from_numpy(memory)                 # what an allocator does with the memory of a model that is gone
    del first
    memory += 1
    second.add_(1)                                    # the same version as the first one had
    assert second.data_ptr() == address and torch.equal(moe_ops._mx_weight(second)[0], second) and len(made) == 3
    del second
    assert len(moe_ops._MX_WEIGHTS) == kept - 1
