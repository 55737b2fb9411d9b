"""GPU parity of the RWKV-7 inference kernels (head size 64, fp32 arithmetic) against the fp64 oracle at the lengths and
unit counts where their forms change: one token, parts of a 16-token stage, and 1, 2 or 4 blocks per unit."""
import pytest
import torch

from oracle import wkv_oracle as O
from tests import helpers as Hh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,T,H", [(3, 1, 5), (1, 2, 3), (2, 15, 3), (1, 17, 38), (2, 33, 2), (3, 47, 37)])
def test_state_update(dtype, B, T, H):
    import rwkv_cuda_b200 as R
    N, names = 64, ("r", "w", "k", "v", "a", "b")
    inp = Hh.v7_inputs(B, T, H, N, seed=T)
    y64, sT64 = O.wkv7(*(inp[n].to(dtype).double() for n in names), H, s0=inp["s0"].double())
    state = inp["s0"].cuda()
    y = torch.full((B, T, H, N), float("nan"), dtype=dtype, device="cuda")
    R.ops.wkv7_state_update(state, *(inp[n].to(dtype).cuda().view(B, T, H, N).contiguous() for n in names), y)
    Hh.assert_close(y.view(B, T, H * N), y64, Hh.tol_for(dtype), "y")
    Hh.assert_close(state, sT64, 1e-5, "state")   # fp32 whatever the activations are
