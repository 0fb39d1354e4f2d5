"""Steps whose scratch memory finds no room run in the form that needs none."""
import gc
from contextlib import contextmanager
from types import SimpleNamespace

import pytest
import torch

from mini_llama_cpp_release_b200 import kernels
from mini_llama_cpp_release_b200.kernels import bindings

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@contextmanager
def room_for(n_bytes):
    """This process may allocate n_bytes more than it has now."""
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(DEV).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved(DEV) + n_bytes) / total, DEV)
    try:
        yield
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, DEV)


def test_a_prompt_through_a_memory_walks_where_its_chunks_find_no_room():
    H, dim, vdim, n = 40, 256, 256, 1024                  # outputs of 42 MB; chunks of 178 MB
    g = torch.Generator().manual_seed(5)
    x = torch.randn(n, 2 * H * dim + 2 * H * vdim, generator=g).to(DEV)
    decay, gain = torch.linspace(0.5, 1.0, H, device=DEV), torch.ones(H * vdim, device=DEV)
    step = SimpleNamespace(n_seqs=1, n_tokens=n, max_q_len=n, cu_seqlens=torch.tensor([0, n], dtype=torch.int32, device=DEV),
                           slots=torch.zeros(1, dtype=torch.int32, device=DEV))
    plan = bindings._head_decay_plan(step, n, H, dim, vdim, DEV)
    assert plan[2] is not None and plan[2].numel() * 4 > 170e6
    del plan

    def run():
        rows, out, state = x.clone(), torch.empty(n, H * vdim, device=DEV), torch.zeros(1, H * dim * vdim, device=DEV)
        return lambda: (kernels.decay_attention(rows, 0, 2 * H * dim + H * vdim, decay, gain, 1e-5, 1.0, state, step, H, dim, vdim, out), out, state)
    _, want, state = run()()
    call = run()
    with room_for(100 << 20):
        _, got, state2 = call()
        torch.cuda.synchronize()
    # float32 sums of up to 256 and 64 products in another order
    assert float((got - want).norm() / want.norm()) <= 1e-5 and float((state2 - state).norm() / state.norm()) <= 1e-5


def test_a_float32_product_runs_in_fewer_blocks_where_its_chunks_find_no_room():
    x, w = torch.randn(256, 896, device=DEV), torch.randn(9728, 896, device=DEV)
    want, got = torch.empty(256, 9728, device=DEV), torch.empty(256, 9728, device=DEV)
    kernels.linear_simt(x, w, want)
    lib = bindings.core()
    assert lib.mlc_linear_simt_scratch_floats(x.data_ptr(), 0, w.data_ptr(), 0, 256, 9728, 896, 148) * 4 > 35e6
    with room_for(20 << 20):
        kernels.linear_simt(x, w, got)
        torch.cuda.synchronize()
    assert torch.equal(got, want)
