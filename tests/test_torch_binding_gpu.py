"""flash_train.torch.gemm on a device: the reference's Python test
(tests/python/torch_gemm_test.py:15-71 there), case for case."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPE_GRID = [(1, 1, 1), (3, 4, 2), (16, 16, 16), (64, 48, 32), (129, 65, 17), (33, 257, 65), (256, 128, 64)]


@pytest.fixture(scope="module")
def binding(native_library):
    if not torch.cuda.is_available():
        pytest.fail("the GPU tests need a CUDA device")
    from conftest import load_build_module

    load_build_module().build_torch_binding(verbose=False)
    torch.backends.cuda.matmul.allow_tf32 = False
    import flash_train.torch

    return flash_train.torch


def make_inputs(shape=(128, 64, 96)):
    generator = torch.Generator(device="cuda").manual_seed(7)
    m, k, n = shape
    a = torch.randn(m, k, device="cuda", generator=generator)
    b = torch.randn(k, n, device="cuda", generator=generator)
    c = torch.randn(m, n, device="cuda", generator=generator)
    return a, b, c


@pytest.mark.parametrize("shape", SHAPE_GRID)
def test_gemm_matches_matmul(binding, shape):
    a, b, c = make_inputs(shape)
    d = binding.gemm(a, b, c, alpha=1.5, beta=0.25)
    torch.testing.assert_close(d, 1.5 * (a @ b) + 0.25 * c, rtol=1e-4, atol=1e-3)


def test_gemm_without_c_and_defaults(binding):
    a, b, _ = make_inputs()
    torch.testing.assert_close(binding.gemm(a, b, alpha=1.5), 1.5 * (a @ b), rtol=1e-4, atol=1e-3)
    torch.testing.assert_close(binding.gemm(a, b), a @ b, rtol=1e-4, atol=1e-3)


def test_runs_on_the_current_stream(binding):
    a, b, _ = make_inputs((512, 256, 384))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        d = binding.gemm(a, b)
    side.synchronize()
    torch.testing.assert_close(d, a @ b, rtol=1e-4, atol=1e-3)


def test_rejections_raise_runtime_error(binding):
    a, b, _ = make_inputs()
    with pytest.raises(RuntimeError):
        binding.gemm(a, torch.randn(3, 3, device="cuda"))
    with pytest.raises(RuntimeError):
        binding.gemm(a.cpu(), b)
    with pytest.raises(RuntimeError):
        binding.gemm(a.to(torch.float64), b)
    with pytest.raises(RuntimeError):
        binding.gemm(a.t(), b)  # not contiguous: rejected by the binding, as in the reference


def test_a_workspace_the_allocator_refuses_is_not_asked_for_on_every_call(binding):
    """With too little memory for the prepared form's workspace the result is that of the form without it, and the allocator,
    which gives back all that it caches at each refusal, is asked once for many calls, whatever their addresses."""
    m = k = n = 2048
    generator = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(m, k, device="cuda", generator=generator)
    b = torch.randn(k, n, device="cuda", generator=generator)
    full = binding.gemm(a, b)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    out_bytes = 4 * m * n  # the prepared form's workspace takes more than two of these; two and a half are left
    total = torch.cuda.get_device_properties(a.device).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 2.5 * out_bytes) / total)
    try:
        before = torch.cuda.memory_stats()["num_alloc_retries"]
        lean = None
        for _ in range(20):
            lean = binding.gemm(a, b)  # the last result is still held: addresses alternate
        torch.cuda.synchronize()
        refusals = torch.cuda.memory_stats()["num_alloc_retries"] - before
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert 1 <= refusals <= 3  # one for each size of the Plan's workspaces
    assert not torch.equal(full, lean), "the prepared form ran after all"
    torch.testing.assert_close(lean, a @ b, rtol=1e-4, atol=1e-3)
    for _ in range(80):  # memory is back: the prepared form is found again
        last = binding.gemm(a, b)
    assert torch.equal(last, full)
