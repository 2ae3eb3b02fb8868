"""Forward parity on the GPU, called through the C ABI: values bit-exact (torch.equal equates
+0/-0, the one place where hardware max and torch.max may differ), indices exactly equal,
lowest k on ties -- against the stored reference outputs and against the C oracle."""
import numpy as np
import pytest
import torch

import capi
from conftest import golden_names, load_golden
from oracle import c_oracle

pytestmark = pytest.mark.gpu

IDX_VARIANTS = [-2, 0, 1, 2, 3, 4, 5, 6, 7]   # -2 = any-shape kernel, 0.. = tiled TMA configurations


def _check_forward(a_np, b_np, y_ref, imax_ref, imin_ref, dev, variant, layout, bias_np=None):
    a = torch.from_numpy(a_np).to(dev)
    b_host = np.ascontiguousarray(b_np.T) if layout == capi.NK else b_np
    b = torch.from_numpy(b_host).to(dev)
    bias = None if bias_np is None else torch.from_numpy(bias_np).to(dev)
    capi.set_variant(True, variant)
    capi.set_variant(False, variant)
    try:
        y, imax, imin = capi.forward(a, b, layout, bias=bias)
        yv, _, _ = capi.forward(a, b, layout, bias=bias, want_idx=False)
    finally:
        capi.set_variant(True, -1)
        capi.set_variant(False, -1)
    assert capi.device_flag_ok()
    y_ref_t = torch.from_numpy(y_ref)
    assert torch.equal(imax.cpu().long(), torch.from_numpy(imax_ref)), "argmax differs"
    assert torch.equal(imin.cpu().long(), torch.from_numpy(imin_ref)), "argmin differs"
    for got in (y.cpu(), yv.cpu()):
        assert torch.equal(got, y_ref_t), "values differ"
        nz = y_ref_t != 0
        assert torch.equal(got[nz].view(torch.int32), y_ref_t[nz].view(torch.int32))


@pytest.mark.parametrize("layout", [capi.KN, capi.NK])
@pytest.mark.parametrize("variant", IDX_VARIANTS)
@pytest.mark.parametrize("name", [n for n in golden_names() if not n.startswith("blend")])
def test_golden_forward(name, variant, layout, cuda):
    g = load_golden(name)
    _check_forward(g["a"], g["b"], g["y"], g["argmax"], g["argmin"], cuda, variant, layout, g.get("bias"))


@pytest.mark.parametrize("variant", [-2, 0])
def test_golden_blend(variant, cuda):
    """(1-beta)*mam + beta*(a@b) + bias through the fused epilogue; the dense term is supplied, so
    the only differences from the reference are fp32 re-association of three terms."""
    g = load_golden("blend_40x64x48")
    a, b = torch.from_numpy(g["a"]).to(cuda), torch.from_numpy(g["b"]).to(cuda)
    beta = float(g["beta"])
    dense = (a.double() @ b.double()).float()
    capi.set_variant(True, variant)
    try:
        y, imax, imin = capi.forward(a, b, capi.KN, bias=torch.from_numpy(g["bias"]).to(cuda), dense=dense,
                                     blend=True, alpha=1 - beta, beta=beta)
    finally:
        capi.set_variant(True, -1)
    assert torch.equal(imax.cpu().long(), torch.from_numpy(g["argmax"]))
    assert torch.equal(imin.cpu().long(), torch.from_numpy(g["argmin"]))
    np.testing.assert_allclose(y.cpu().numpy(), g["y"], rtol=1e-5, atol=1e-5)


SHAPES = [(300, 260, 200), (1, 64, 1), (65, 4, 63), (128, 32, 128), (257, 96, 129), (1000, 768, 520),
          (130, 36, 70), (64, 2048, 64), (513, 100, 257)]


@pytest.mark.parametrize("variant", IDX_VARIANTS)
@pytest.mark.parametrize("shape", SHAPES)
def test_random_against_c_oracle(shape, variant, cuda):
    M, K, N = shape
    g = torch.Generator().manual_seed(M * 7 + K * 3 + N)
    a = torch.randn(M, K, generator=g)
    w = torch.randn(N, K, generator=g) * K ** -0.5
    y_ref, imax_ref, imin_ref = c_oracle.forward(a.numpy(), w.numpy(), b_is_nk=True)
    _check_forward(a.numpy(), np.ascontiguousarray(w.numpy().T), y_ref, imax_ref, imin_ref, cuda, variant, capi.NK)


@pytest.mark.parametrize("variant", IDX_VARIANTS)
def test_ties_zeros_and_signs(variant, cuda):
    """Integer-valued operands, ReLU'd activations and pruned weights: most products tie (many at
    +0/-0), so the index is decided by the lowest-k rule in every chunk and across chunks."""
    g = torch.Generator().manual_seed(11)
    M, K, N = 200, 416, 136
    a = torch.relu(torch.randint(-2, 3, (M, K), generator=g).float())
    w = torch.randint(-2, 3, (N, K), generator=g).float() * (torch.rand(N, K, generator=g) > 0.5)
    a[5] = 0  # a row of zeros: every product is +-0, argmax = argmin = 0
    w[7] = 0
    y_ref, imax_ref, imin_ref = c_oracle.forward(a.numpy(), w.numpy(), b_is_nk=True)
    assert (imax_ref[5] == 0).all() and (imin_ref[:, 7] == 0).all()
    _check_forward(a.numpy(), np.ascontiguousarray(w.numpy().T), y_ref, imax_ref, imin_ref, cuda, variant, capi.NK)


SLICED_SHAPES = [(1, 4, 1), (7, 260, 129), (8, 768, 300), (33, 1028, 65), (65, 36, 130), (130, 2084, 70)]


@pytest.mark.parametrize("variant", range(8, 20))
@pytest.mark.parametrize("shape", SLICED_SHAPES)
def test_sliced_forms(shape, variant, cuda):
    """Every tile and cluster size of the sliced kernel at ragged tiles, fewer chunks than slices and a ragged last
    chunk; half of the operands are small integers, so ties cross chunks and slices.  Bit for bit, the oracle's."""
    M, K, N = shape
    g = torch.Generator().manual_seed(M * 5 + K * 11 + N)
    a = torch.randn(M, K, generator=g)
    w = torch.randn(N, K, generator=g) * K ** -0.5
    a[: M // 2] = torch.randint(-2, 3, (M // 2, K), generator=g).float()
    w[: N // 2] = torch.randint(-2, 3, (N // 2, K), generator=g).float()
    y_ref, imax_ref, imin_ref = c_oracle.forward(a.numpy(), w.numpy(), b_is_nk=True)
    _check_forward(a.numpy(), np.ascontiguousarray(w.numpy().T), y_ref, imax_ref, imin_ref, cuda, variant, capi.NK)


@pytest.mark.parametrize("layout", [capi.KN, capi.NK])
@pytest.mark.parametrize("shape", [(64, 257, 64), (131, 1001, 129), (1, 2047, 600), (700, 33, 515), (2100, 70, 1030),
                                   (5000, 133, 1030), (38100, 245, 70), (38100, 27, 70)])
def test_ragged_k(shape, layout, cuda):
    """K that is no multiple of 4, large enough for the padded copies: the automatic choice (any-shape kernel, or copies
    and the sliced or, beyond 592 tiles, the tiled kernel and the resolver) against the oracle, with ties at the last
    (repeated) element."""
    M, K, N = shape
    g = torch.Generator().manual_seed(M + K * 3 + N)
    a = torch.randn(M, K, generator=g)
    w = torch.randn(N, K, generator=g) * K ** -0.5
    a[::2], w[::2] = a[::2].round(), w[::2].round()
    a[0, -1], w[0, -1], w[-1, -1] = 40.0, 40.0, -40.0
    y_ref, imax_ref, imin_ref = c_oracle.forward(a.numpy(), w.numpy(), b_is_nk=True)
    assert imax_ref[0, 0] == K - 1
    _check_forward(a.numpy(), np.ascontiguousarray(w.numpy().T), y_ref, imax_ref, imin_ref, cuda, -1, layout)


@pytest.mark.parametrize("layout", [capi.KN, capi.NK])
@pytest.mark.parametrize("variant", [-2, -1, 0, 2, 8, 13, 19])   # any-shape, by size, tiled + resolver, sliced
@pytest.mark.parametrize("shape", [(1500, 5, 150), (900, 9, 140), (38000, 9, 100), (400, 25, 131), (300, 27, 130),
                                   (300, 33, 130), (260, 36, 130), (131, 100, 129), (50, 36, 60)])
def test_nan_and_infinite_products(shape, variant, layout, cuda):
    """Rows and weights of NaN and infinities on every route: indices inside [0, K) and the oracle's, 0 where no
    product is above -inf (max) or below +inf (min)."""
    M, K, N = shape
    nan, inf = float("nan"), float("inf")
    g = torch.Generator().manual_seed(M + K + N)
    a, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    a[0], a[1], a[2], a[3] = nan, inf, -inf, 0.0
    a[4, : K // 2], a[4, K // 2:] = nan, -inf
    a[5, : K // 2], a[5, K // 2:] = nan, inf
    a[6, K - 1], a[-1] = inf, nan
    w[0], w[1], w[2], w[3], w[4, 0], w[-1] = w[0].abs(), -w[1].abs(), 0.0, nan, -inf, nan
    y_ref, imax_ref, imin_ref = c_oracle.forward(a.numpy(), w.numpy(), b_is_nk=True)
    assert (imax_ref[0] == 0).all() and (imin_ref[:, 3] == 0).all()
    b = (w.T.contiguous() if layout == capi.KN else w).to(cuda)
    capi.set_variant(True, variant)
    try:
        y, imax, imin = capi.forward(a.to(cuda), b, layout)
    finally:
        capi.set_variant(True, -1)
    assert capi.device_flag_ok()
    assert torch.equal(imax.cpu().long(), torch.from_numpy(imax_ref))
    assert torch.equal(imin.cpu().long(), torch.from_numpy(imin_ref))
    assert np.array_equal(y.cpu().numpy(), y_ref, equal_nan=True)


@pytest.mark.parametrize("layout", [capi.KN, capi.NK])
@pytest.mark.parametrize("variant", [0, 2, 5, 7, 8, 13, 18])
@pytest.mark.parametrize("shape", [(300, 29, 150), (131, 1001, 129), (65, 258, 130)])
def test_ragged_k_in_every_kernel(shape, variant, layout, cuda):
    """Padded copies into the tiled and sliced configurations: rows of 1, 2 and 3 elements beyond a multiple of 4, ties."""
    M, K, N = shape
    g = torch.Generator().manual_seed(M + K * 3 + N)
    a, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    a[::2], w[::2] = a[::2].round(), w[::2].round()
    a[0, -1], w[0, -1], w[-1, -1] = 40.0, 40.0, -40.0
    y_ref, imax_ref, imin_ref = c_oracle.forward(a.numpy(), w.numpy(), b_is_nk=True)
    _check_forward(a.numpy(), np.ascontiguousarray(w.numpy().T), y_ref, imax_ref, imin_ref, cuda, variant, layout)


def test_ragged_k_without_memory_for_the_copies(cuda):
    """The padded copies are as large as the operands; where they do not fit any more the call still runs."""
    from mamtorch_b200 import _lib

    M, K, N = 150000, 1001, 8
    g = torch.Generator(device=cuda).manual_seed(3)
    x, w = torch.randn(M, K, generator=g, device=cuda), torch.randn(N, K, generator=g, device=cuda)
    need = _lib.lib().mam_fwd_workspace_bytes(M, K, N, capi.NK, 0)
    op = lambda: torch.ops.mamtorch_b200.linear_forward(x, w, None, None, 1.0, 0.0, False)[0]
    y = op()
    torch.cuda.empty_cache()
    limit = torch.cuda.memory_reserved() + need // 2
    assert need > x.numel() * 4
    torch.cuda.set_per_process_memory_fraction(limit / torch.cuda.get_device_properties(0).total_memory)
    try:
        short = op()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(short, y)


@pytest.mark.parametrize("shape,status", [((8, 64, 100), 0), ((1, 1024, 4095), 0), ((64, 36, 64), 3), ((131, 1001, 129), 0)])
def test_column_major_weight_without_workspace(shape, status, cuda):
    """b[K,N] and no scratch: small products and K % 4 != 0 run in the any-shape kernel, others are refused."""
    from mamtorch_b200 import _lib

    M, K, N = shape
    g = torch.Generator().manual_seed(M + K + N)
    a, b = torch.randn(M, K, generator=g).to(cuda), torch.randn(K, N, generator=g).to(cuda)
    y = torch.empty(M, N, device=cuda)
    imax, imin = torch.empty_like(y, dtype=torch.int32), torch.empty_like(y, dtype=torch.int32)
    st = _lib.lib().mam_fwd_f32(capi._ptr(a), capi._ptr(b), capi.KN, None, None, 0, 1.0, 0.0, capi._ptr(y),
                                capi._ptr(imax), capi._ptr(imin), M, K, N, None, 0, capi._stream())
    assert st == status
    if status == 0:
        y_ref, imax_ref, imin_ref = c_oracle.forward(a.cpu().numpy(), np.ascontiguousarray(b.cpu().numpy().T), b_is_nk=True)
        assert torch.equal(y.cpu(), torch.from_numpy(y_ref))
        assert torch.equal(imax.cpu().long(), torch.from_numpy(imax_ref))
        assert torch.equal(imin.cpu().long(), torch.from_numpy(imin_ref))


RESOLVER_SHAPES = [(300, 260, 200), (65, 4, 63), (129, 2080, 131), (257, 96, 129), (520, 2500, 140), (64, 2048, 64),
                   (1, 64, 1), (200, 416, 136)]


@pytest.mark.parametrize("form", [0, 1])   # tiled, thread per output
@pytest.mark.parametrize("shape", RESOLVER_SHAPES)
def test_resolver_forms(shape, form, cuda):
    """Both forms of the chunk-id -> index step, forced whatever the shape, against the C oracle; half of the
    operands are small integers so that ties inside and across chunks are decided by the lowest-k rule."""
    from mamtorch_b200 import _lib

    M, K, N = shape
    g = torch.Generator().manual_seed(M * 5 + K * 11 + N)
    a = torch.randn(M, K, generator=g)
    w = torch.randn(N, K, generator=g) * K ** -0.5
    a[: M // 2] = torch.randint(-2, 3, (M // 2, K), generator=g).float()
    w[: N // 2] = torch.randint(-2, 3, (N // 2, K), generator=g).float()
    y_ref, imax_ref, imin_ref = c_oracle.forward(a.numpy(), w.numpy(), b_is_nk=True)
    _lib.check(_lib.lib().mam_tune_set(2, form), "resolver form")
    try:
        _check_forward(a.numpy(), np.ascontiguousarray(w.numpy().T), y_ref, imax_ref, imin_ref, cuda, 0, capi.NK)
    finally:
        _lib.lib().mam_tune_set(2, 0)


def test_unaligned_views_take_the_any_shape_path(cuda):
    """Pointers that are not 16-byte aligned cannot be described to TMA; the call must still work."""
    g = torch.Generator().manual_seed(5)
    M, K, N = 70, 64, 66
    abuf = torch.randn(M * K + 1, generator=g)
    wbuf = torch.randn(N * K + 1, generator=g)
    a_np, w_np = abuf[1:].view(M, K).numpy(), wbuf[1:].view(N, K).numpy()
    y_ref, imax_ref, imin_ref = c_oracle.forward(a_np, w_np, b_is_nk=True)
    a = abuf.to(cuda)[1:].view(M, K)
    w = wbuf.to(cuda)[1:].view(N, K)
    assert a.data_ptr() % 16 != 0
    y, imax, imin = capi.forward(a, w, capi.NK)
    assert torch.equal(y.cpu(), torch.from_numpy(y_ref))
    assert torch.equal(imax.cpu().long(), torch.from_numpy(imax_ref))
    assert torch.equal(imin.cpu().long(), torch.from_numpy(imin_ref))


def test_full_size_properties(cuda):
    """At a benchmark-sized problem (ViT-B/16 MLP layer 1: 12608 x 768 -> 3072) the oracle is too slow
    for a full comparison; check properties that hold at any size instead:
      * y equals the sum of the two products at the returned indices (bit for bit);
      * no product beats them (checked on a random sample of rows against the C oracle);
      * values-only and index-producing kernels agree; two runs are bit-identical."""
    M, K, N = 12608, 768, 3072
    g = torch.Generator().manual_seed(0)
    a = torch.randn(M, K, generator=g).to(cuda)
    w = (torch.randn(N, K, generator=g) * K ** -0.5).to(cuda)
    y, imax, imin = capi.forward(a, w, capi.NK)
    yv, _, _ = capi.forward(a, w, capi.NK, want_idx=False)
    y2, imax2, imin2 = capi.forward(a, w, capi.NK)
    assert capi.device_flag_ok()
    assert torch.equal(y, yv) and torch.equal(y, y2) and torch.equal(imax, imax2) and torch.equal(imin, imin2)
    assert int(imax.min()) >= 0 and int(imax.max()) < K and int(imin.min()) >= 0 and int(imin.max()) < K
    rows = torch.arange(M, device=cuda)[:, None].expand(M, N)
    cols = torch.arange(N, device=cuda)[None, :].expand(M, N)
    pmax = a[rows, imax.long()] * w[cols, imax.long()]
    pmin = a[rows, imin.long()] * w[cols, imin.long()]
    assert torch.equal(y, pmax + pmin)
    sample = torch.randint(0, M, (24,), generator=g)
    y_ref, imax_ref, imin_ref = c_oracle.forward(a[sample.to(cuda)].cpu().numpy(), w.cpu().numpy(), b_is_nk=True)
    assert torch.equal(y[sample.to(cuda)].cpu(), torch.from_numpy(y_ref))
    assert torch.equal(imax[sample.to(cuda)].cpu().long(), torch.from_numpy(imax_ref))
    assert torch.equal(imin[sample.to(cuda)].cpu().long(), torch.from_numpy(imin_ref))
