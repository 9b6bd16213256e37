"""rt.log_mse on the GPU against the same formula in FP64 tensor operations: value, gradient and
higher derivatives, the sizes around its one-block and many-block kernels, the values it leaves
out, and the forms that keep the tensor operations."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
rt = pytest.importorskip("ragnar_gb300.torch_ext")


def _formula(S, T, floor=1e-12):
    m = (S > floor * S.detach().max()) & (T > floor * T.max())
    d = torch.log(torch.where(m, S, torch.ones_like(S))) - torch.log(torch.where(m, T, torch.ones_like(T)))
    return (d * d * m).sum() / m.sum().clamp(min=1)


def _spectra(shape, seed, dev):
    rng = np.random.default_rng(seed)
    S = 10.0 ** rng.uniform(-9.0, 6.0, shape)
    T = S * 10.0 ** rng.uniform(-1.0, 1.0, shape)
    return (torch.from_numpy(S.astype(np.float32)).to(dev).requires_grad_(True),
            torch.from_numpy(T.astype(np.float32)).to(dev))


@pytest.mark.parametrize("shape", [(1,), (31,), (512,), (1025,), (8192,), (8193,), (1024, 200), (3, 1_000_003)])
def test_value_and_gradient(gpu, shape):
    """A term's error is that of two FP32 logarithms of magnitude below 21 (2.5e-6 each) against
    |d| up to 2.3: far below 1e-5 of the mean, and 1e-5 of the largest gradient."""
    S, T = _spectra(shape, sum(shape), gpu)
    loss = rt.log_mse(S, T)
    (g,) = torch.autograd.grad(loss, S)
    S64 = S.detach().double().requires_grad_(True)
    want = _formula(S64, T.double())
    (g64,) = torch.autograd.grad(want, S64)
    assert loss.shape == () and loss.dtype == torch.float32 and g.shape == S.shape
    assert abs(float(loss) - float(want)) <= 1e-5 * float(want)
    rel = torch.abs(g.double() - g64) * S64.detach()  # dL/d ln S
    assert float(rel.max()) <= 1e-5 * float((g64 * S64.detach()).abs().max())


def test_higher_derivatives(gpu):
    S, T = _spectra((64,), 5, gpu)
    with torch.no_grad():
        S.copy_(torch.rand(64, device=gpu) + 0.5)
        T = torch.rand(64, device=gpu) + 0.5
    S64 = S.detach().double().requires_grad_(True)
    got, want = rt.log_mse(S * 1.5, T), _formula(S64 * 1.5, T.double())
    for order in range(4):
        (got,) = torch.autograd.grad((got * got).sum() if order else got, S, create_graph=True)
        (want,) = torch.autograd.grad((want * want).sum() if order else want, S64, create_graph=True)
        assert float((got.double() - want).abs().max()) <= 1e-4 * float(want.abs().max())


@pytest.mark.parametrize("case", ["nan", "inf", "zeros", "negative", "floor"])
def test_left_out_values(gpu, case):
    S, T = _spectra((700,), 9, gpu)
    floor = 1e-3 if case == "floor" else 1e-12
    with torch.no_grad():
        if case == "nan":
            S[3] = float("nan")
        elif case == "inf":
            T[5] = float("inf")
        elif case == "zeros":
            S[::2] = 0.0
            T[::3] = 0.0
        elif case == "negative":
            S[::5] = -1.0
    ref = S.detach().clone().requires_grad_(True)
    got, want = rt.log_mse(S, T, floor), _formula(ref, T, floor)
    (g,), (h,) = torch.autograd.grad(got, S), torch.autograd.grad(want, ref)
    assert torch.allclose(got, want, rtol=1e-5, equal_nan=True)
    assert torch.equal(g == 0, h == 0) and torch.allclose(g, h, rtol=1e-4, atol=0, equal_nan=True)


def test_forms_that_keep_the_tensor_operations(gpu):
    """A target that takes a gradient, FP64, strided and broadcast spectra, vmap and forward mode;
    and a spectrum that is changed in place between loss and backward."""
    S, T = _spectra((6, 40), 3, gpu)
    Tg = T.clone().requires_grad_(True)
    rt.log_mse(S, Tg).backward()
    assert Tg.grad is not None and S.grad is not None
    assert rt.log_mse(S.double(), T.double()).dtype == torch.float64
    assert torch.allclose(rt.log_mse(S.t(), T.t()), rt.log_mse(S, T))
    assert torch.allclose(rt.log_mse(S[:1], T), _formula(S[:1], T))
    v = torch.func.vmap(rt.log_mse)(S.detach(), T)
    assert torch.allclose(v, torch.stack([_formula(a, b) for a, b in zip(S.detach(), T)]), rtol=1e-5)
    _, t = torch.func.jvp(lambda s: rt.log_mse(s, T), (S.detach(),), (S.detach(),))
    (g,) = torch.autograd.grad(rt.log_mse(S, T), S)
    assert torch.allclose(t, (g * S.detach()).sum(), rtol=1e-4)
    y = S * 1.0
    loss = rt.log_mse(y, T)
    y.mul_(2.0)
    (h,) = torch.autograd.grad(loss, S)
    assert torch.allclose(h, g, rtol=1e-5)
    total = rt.log_mse(S, T)
    total += 1.0
    (h,) = torch.autograd.grad(total, S)
    assert torch.equal(h, g)


def test_negated_view(gpu):
    """The imaginary part of a conjugate is a view whose memory holds the opposite values."""
    z = torch.tensor([1.0 - 2.0j], device=gpu)
    S, T = z.conj().imag, torch.tensor([3.0], device=gpu)
    assert S.is_neg() and S.is_contiguous() and S.dtype == torch.float32
    assert abs(float(rt.log_mse(S, T)) - np.log(2.0 / 3.0) ** 2) <= 1e-6


@pytest.mark.parametrize("scale", [1e-24, 1e-22, 1e-12, 1e12, 1e20, 1e22, 1e24])
def test_hessian_vector_product_far_from_one(gpu, scale):
    """A vector of the spectrum's own size: the product is about 1 / S, although 1 / S^2 is not a float.
    Its terms are products of six FP32 factors with |d| up to 2.3, and differ by at most that factor
    from the largest of them: 1e-5 of it."""
    rng = np.random.default_rng(8)
    s = scale * 10.0 ** rng.uniform(-0.5, 0.5, 64)
    t = s * 10.0 ** rng.uniform(-1.0, 1.0, 64)
    v = s * rng.uniform(0.5, 1.5, 64)
    S = torch.from_numpy(s.astype(np.float32)).to(gpu).requires_grad_(True)
    T, V = (torch.from_numpy(x.astype(np.float32)).to(gpu) for x in (t, v))
    S64 = S.detach().double().requires_grad_(True)
    (g,) = torch.autograd.grad(rt.log_mse(S, T), S, create_graph=True)
    (h,) = torch.autograd.grad((g * V).sum(), S)
    (g64,) = torch.autograd.grad(_formula(S64, T.double()), S64, create_graph=True)
    (h64,) = torch.autograd.grad((g64 * V.double()).sum(), S64)
    assert float((h.double() - h64).abs().max()) <= 1e-5 * float(h64.abs().max())


def test_gradient_of_spectra_near_the_smallest_float(gpu):
    """2 (ln S - ln T) / S is above the float range where the gradient, its share of 512 values, is not."""
    rng = np.random.default_rng(10)
    S = torch.from_numpy((3e-38 * rng.uniform(1.0, 9.0, 512)).astype(np.float32)).to(gpu).requires_grad_(True)
    T = (S.detach() * 1e4).contiguous()
    (g,) = torch.autograd.grad(rt.log_mse(S, T), S)
    S64 = S.detach().double().requires_grad_(True)
    (g64,) = torch.autograd.grad(_formula(S64, T.double()), S64)
    assert float(g64.abs().max()) < 3e38 and float((2 * torch.log(S64 / T.double()) / S64).abs().max()) > 3.5e38
    assert float((g.double() - g64).abs().max()) <= 1e-5 * float(g64.abs().max())
