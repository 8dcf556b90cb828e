"""Operands written by the very launch in front of the call that reads them.  Kernels of this library start while their
predecessor drains and may fetch weights before they wait for it; a call made on its own has to see what the call in front of
it wrote all the same.  Each case queues a long launch, the writer and the reader without a synchronisation and compares with
the reader alone afterwards: equal bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from glm_asr_stack_b200 import ops as _ops
    yield _ops
    assert _ops.status() == 0


def check(ops, write, read, trials=6):
    busy = torch.randn((20000, 2048), device="cuda").to(torch.bfloat16)
    one = torch.ones(2048, dtype=torch.bfloat16, device="cuda")
    for t in range(trials):
        write(0)                                  # other contents first
        read()
        torch.cuda.synchronize()
        for _ in range(3):
            ops.rmsnorm(busy, one, out=busy)      # keeps the device behind the host
        write(1 + t)
        got = read()
        torch.cuda.synchronize()
        assert torch.equal(got.view(torch.int16), read().view(torch.int16)), t


@pytest.mark.parametrize("M", [1, 8, 19, 64])
@pytest.mark.parametrize("native", [True, False])
def test_fp4_weight_quantised_in_front_of_its_linear(ops, M, native):
    from glm_asr_stack_b200 import _lib
    lib = _lib.load()
    N = K = 2048
    packed = torch.empty((N, K // 2), dtype=torch.uint8, device="cuda")
    scales = torch.empty((N, K // 16), dtype=torch.uint8, device="cuda")
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (packed, scales)]
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
    src = [torch.randn((N, K), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(7)]

    def write(i):
        lib.glmasr_fp4_forget(ptr[1])             # cached state of the weight that is about to change
        assert lib.glmasr_quantize_bf16_to_fp4(ptr[0], ptr[1], ctypes.c_void_p(src[i].data_ptr()), None, 0.002, N, K) == 0

    def read():
        if not native:
            return ops.fp4_linear(x, packed, scales, 0.002)
        out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        assert ops.nvfp4_linear(out, x, packed, scales, 0.002, 0.002) == 0
        return out

    check(ops, write, read)


@pytest.mark.parametrize("M", [1, 19, 600])
def test_bf16_weight_computed_in_front_of_its_linear(ops, M):
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, 512), generator=gen, device="cuda").to(torch.bfloat16)
    src = [torch.randn((1024, 512), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(7)]
    one = torch.ones(512, dtype=torch.bfloat16, device="cuda")
    w = torch.empty((1024, 512), dtype=torch.bfloat16, device="cuda")
    check(ops, lambda i: ops.rmsnorm(src[i], one, out=w), lambda: ops.bf16_linear(x, w))


@pytest.mark.parametrize("rows", [1, 200, 4000])
def test_layernorm_weights_computed_in_front_of_it(ops, rows):
    dim = 1280
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, dim), generator=gen, device="cuda").to(torch.bfloat16)
    src = [torch.randn((2048, dim), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(7)]
    one = torch.ones(dim, dtype=torch.bfloat16, device="cuda")
    params = torch.empty((2048, dim), dtype=torch.bfloat16, device="cuda")
    # the last rows of a norm over many: what its last CTAs write
    check(ops, lambda i: ops.rmsnorm(src[i], one, out=params), lambda: ops.layernorm(x, params[2046], params[2047]))
