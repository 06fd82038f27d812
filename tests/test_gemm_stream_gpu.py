"""The streamed product of a decode step (``gemm_stream.cu``) against the plain 32-bit product of the same operands: one
chunk of features an SM and several, row tiles that are full, ragged and a single row, ragged last stages, rings that hold everything
and rings that turn, one and two token tiles, every epilogue, the norm before the product, and operands that it refuses."""
import pytest
import torch

from gpu_util import assert_close
from torch_ops import TorchOps

from nanoinfer_b200.config import KernelOptions

pytestmark = pytest.mark.gpu
REF = TorchOps()
BF16 = torch.bfloat16


@pytest.fixture(scope="module")
def K():
    from nanoinfer_b200.csrc.lib import load_kernels
    k = load_kernels().with_options(gemm_route="stream").with_weights_ahead()      # as a model has it
    yield k
    k.check_device_errors()


@pytest.fixture()
def ran(K, monkeypatch):
    """Whether each product that was meant for this kernel was taken by it."""
    taken, plain = [], K._streamed
    monkeypatch.setattr(K, "_streamed", lambda *a: taken.append(plain(*a)) or taken[-1], raising=False)
    return taken


def rnd(shape, seed, scale=1.0, dtype=BF16):
    x = (scale * torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")).to(dtype)
    torch.cuda.synchronize()        # the kernel reads its weights before it waits for the kernel before it: they are nobody's output
    return x


# features an SM: 1, 7 (a tile of its own), 17, 34 (an odd tile over the halves), 64, and 65 (two chunks of 33). From 2,048 k on eight CTAs
# share them: 50 and 64 features each, held whole; two chunks through the ring; the same with a last stretch of k that is shorter
@pytest.mark.parametrize("n,k", [(5, 64), (896, 4864), (1152, 5632), (1536, 2560), (2048, 2304), (1000, 192), (2500, 1536), (4900, 320), (9472, 128), (9500, 704)])
@pytest.mark.parametrize("m", [1, 3, 8, 9, 16])
def test_streamed_sum(K, ran, m, n, k):
    a, w, bias = rnd((m, k), 1), rnd((n, k), 2, k ** -0.5), rnd((n,), 3, dtype=torch.float32)
    out = rnd((m, n), 4, dtype=torch.float32)
    want = a.double() @ w.double().t() + bias.double() + out.double()
    K.linear(a, w, bias, out, "add")
    assert ran == [True]
    assert_close(out, want, torch.float32, "the sum")
    if k > 2048:        # CTAs that share K add up in any order
        return
    whole = torch.zeros(m, n, device="cuda")
    K.linear(a, w, None, whole, "add")
    for i in range(m):      # a row's sums do not depend on the rows beside it
        row = torch.zeros(1, n, device="cuda")
        K.linear(a[i:i + 1], w, None, row, "add")
        assert torch.equal(row[0], whole[i])
    assert ran == [True] * (m + 2)


@pytest.mark.parametrize("inter,k", [(3, 64), (320, 192), (4864, 896), (8960, 1536), (9500, 128)])
@pytest.mark.parametrize("m", [1, 8, 11, 16])
@pytest.mark.parametrize("kind", ["silu", "gelu_tanh", "glu"])
def test_streamed_gated_product(K, ran, m, inter, k, kind):
    a, w = rnd((m, k), 5), rnd((2 * inter, k), 6, k ** -0.5)
    out, ref = torch.empty(m, inter, dtype=BF16, device="cuda"), torch.empty(m, inter, dtype=BF16, device="cuda")
    args = dict(glu=(1.702, 7.0, 1.0)) if kind == "glu" else dict(act=kind)
    K.linear_swiglu(a, w, out, **args)
    assert ran == [True]
    REF.linear_swiglu(a, w, ref, **args)
    assert_close(out, ref, BF16, kind)


def behind_a_norm(K, m, hidden, inter):
    from nanoinfer_b200.parts.base import Runtime
    from nanoinfer_b200.parts.norm import RMSNorm
    x, w = rnd((m, hidden), 7, 3.0, torch.float32), rnd((2 * inter, hidden), 10, hidden ** -0.5)
    return RMSNorm(RMSNorm.spec(hidden, 1e-5, "g"), {"gain": 1.0 + rnd((hidden,), 11, 0.3, torch.float32)}, Runtime(torch.device("cuda"), BF16, K)), x, w


@pytest.mark.parametrize("hidden,inter", [(896, 4864), (64, 100), (1984, 50), (704, 9500)])
@pytest.mark.parametrize("m", [1, 7, 8, 16])
def test_streamed_gated_product_behind_a_norm(K, ran, m, hidden, inter):
    norm, x, w = behind_a_norm(K, m, hidden, inter)
    lazy = norm.lazy(x)
    out, ref = torch.empty(m, inter, dtype=BF16, device="cuda"), torch.empty(m, inter, dtype=BF16, device="cuda")
    K.linear_swiglu(lazy, w, out)
    assert ran == [True] and (lazy.resolved is None) == (m <= 8)        # nobody computed the norm of few tokens
    REF.linear_swiglu(norm.forward(x), w, ref)
    assert_close(out, ref, BF16, "the product behind the norm")


@pytest.mark.parametrize("m,taken", [(9, True), (10, False), (12, False), (16, False)])
def test_activations_that_do_not_fit_go_on_to_another_kernel(K, ran, monkeypatch, m, taken):
    """16-bit rows of 3,584: nine are 64 KB. The norm that was computed for the refused product is the next kernel's operand."""
    monkeypatch.setattr(K, "options", KernelOptions())
    norm, x, w = behind_a_norm(K, m, 3584, 4096)
    lazy = norm.lazy(x)
    out, ref = torch.empty(m, 4096, dtype=BF16, device="cuda"), torch.empty(m, 4096, dtype=BF16, device="cuda")
    K.linear_swiglu(lazy, w, out)
    assert ran == [taken] and lazy.resolved is not None
    REF.linear_swiglu(norm.forward(x), w, ref)
    assert_close(out, ref, BF16, "the product behind the norm")


def test_a_norm_of_more_tokens_than_it_computes_is_refused(K):
    """Asked directly: nothing is launched."""
    import ctypes
    x, w, gain, out = rnd((9, 128), 1, 1.0, torch.float32), rnd((64, 128), 2), rnd((128,), 3, 1.0, torch.float32), torch.zeros(9, 32, dtype=BF16, device="cuda")
    p, i = lambda t: ctypes.c_void_p(t.data_ptr()), ctypes.c_int        # noqa: E731
    for tokens, rc in ((8, 0), (9, 1)):
        got = K._lib.nib_gemm_stream(p(x), p(w), None, p(out), i(tokens), i(32), i(128), i(128), i(32), i(3), i(1), p(gain), ctypes.c_float(1e-5), None, K._stream())
        assert got == rc, tokens
    torch.cuda.synchronize()
    assert bool((out[8] == 0).all())
