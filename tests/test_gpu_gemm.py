"""INT4 g128 GEMM on the tcgen05 tensor cores against the CPU oracle's matmul
(C[m,n] = sum_k f16(A[m,k]/awq[k]) * f16((q-z)s), f32 accumulation, fp16 result)."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests import helpers as H

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# tolerance: same fp16 operands, f32 accumulation in a different order, one fp16 rounding of the result
TOL = 2e-3


@pytest.fixture(scope="module")
def dev():
    from ironmill_b200 import ops
    return ops.Device(0)


def _check(dev, qw, M, seed=0):
    from ironmill_b200 import ops
    x = (H.rng_for("gemm-x", seed).standard_normal((M, qw.K))).astype(np.float16)
    y = ops.matmul_affine(qw.gpu(dev), torch.from_numpy(x).cuda()).cpu().numpy()
    ref = orc.matmul_affine(qw.packed, qw.scales_f16, qw.zps_f16, x, qw.N, qw.K, 128, 4, awq=qw.awq, threads=8)
    err = H.rel_err(y, ref)
    assert err <= TOL, (qw.N, qw.K, M, err)
    return y, ref


@pytest.mark.parametrize("N,K,M", [(128, 128, 16), (256, 512, 32), (384, 1024, 70), (128, 256, 200), (1024, 1024, 129), (640, 384, 1)])
def test_shapes_and_token_tails(dev, N, K, M):
    _check(dev, H.QWeight(N, K, seed=N + M, name="g"), M)


@pytest.mark.parametrize("N,K,M", [(512, 2048, 16), (512, 2048, 64), (384, 1792, 33), (1024, 14336, 16), (200, 1024, 7)])
def test_k_split_for_few_tokens(dev, N, K, M):
    # at most 64 tokens against few 128-row tiles: the grid is cut along K (four slices here; an uneven last slice at
    # K = 1792 = 14 groups; ragged rows at N = 200), the f32 slices are added in order and rounded once
    _check(dev, H.QWeight(N, K, awq=True, seed=N + K + M, name="gk"), M)


@pytest.mark.parametrize("N,K,M", [(256, 512, 32), (384, 1024, 70), (1024, 1024, 129), (512, 2048, 16), (200, 512, 300)])
def test_int8_weights(dev, N, K, M):
    # superblock_matmul_int8 (affine_matmul.metal:155-290): byte codes through the same tensor-core kernel
    qw = H.QWeight(N, K, bits=8, awq=True, seed=N + K + M, name="g8")
    from ironmill_b200 import ops
    x = (H.rng_for("gemm-x8", M).standard_normal((M, K))).astype(np.float16)
    y = ops.matmul_affine(qw.gpu(dev), torch.from_numpy(x).cuda()).cpu().numpy()
    ref = orc.matmul_affine(qw.packed, qw.scales_f16, qw.zps_f16, x, N, K, 128, 8, awq=qw.awq, threads=8)
    assert H.rel_err(y, ref) <= TOL, (N, K, M)


def test_many_token_tiles_of_256(dev):
    # 19 token tiles x 8 row tiles: the 256-token tile (chosen once the grid covers the GPU), a ragged last token tile
    _check(dev, H.QWeight(1024, 512, awq=True, seed=77, name="gt"), 4700)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("N,K,M,awq", [(9480, 128, 129, False), (9472, 384, 257, True), (2376, 640, 1025, True), (2504, 1792, 2047, False), (20000, 256, 300, True)])
def test_cta_pairs(dev, N, K, M, awq, bits):
    # tiles of 256 rows x 128 or 256 tokens: ragged last row tile (N % 256 from 0 to 248), one token more and less than a tile,
    # one to fourteen groups against rings of three and four stages, more tiles than pairs
    from ironmill_b200 import ops
    qw = H.QWeight(N, K, bits=bits, awq=awq, seed=N + M + bits, name="gp")
    qw.zps = qw.zps.copy()
    qw.zps[5::977] += 0.5  # a zero point that is no integer: the f32 path
    qw.zps_f16 = orc.f32_to_f16(qw.zps)
    x = (H.rng_for("gemm-xp", M).standard_normal((M, K))).astype(np.float16)
    y = ops.matmul_affine(qw.gpu(dev), torch.from_numpy(x).cuda()).cpu().numpy()
    ref = orc.matmul_affine(qw.packed, qw.scales_f16, qw.zps_f16, x, N, K, 128, bits, awq=qw.awq, threads=8)
    assert H.rel_err(y, ref) <= TOL, (N, K, M)


def test_awq_and_ragged_rows(dev):
    # N not a multiple of the 128-row CTA tile: the last CTA's spare rows are masked
    _check(dev, H.QWeight(200, 512, awq=True, seed=3, name="ga"), 48)


def test_llama_projection_shape(dev):
    _check(dev, H.QWeight(4096, 4096, awq=True, seed=5, name="gl"), 256)


def test_unusual_zero_points_take_the_f32_path(dev):
    # zero points that are not small integers (possible in a bundle written by another quantiser)
    qw = H.QWeight(256, 256, seed=9, name="gz")
    qw.zps = qw.zps.copy()
    qw.zps[::3] += 0.5
    qw.zps[1::7] = 3000.0
    qw.zps_f16 = orc.f32_to_f16(qw.zps)
    _check(dev, qw, 40)


@pytest.mark.parametrize("awq", [False, True])
@pytest.mark.parametrize("K,M", [(512, 16), (512, 130), (4096, 1200)])
def test_result_over_the_tokens(dev, K, M, awq):
    # out may be x: K split over the grid, whole tiles, CTA pairs with more tiles than pairs (later ones read what earlier ones wrote)
    from ironmill_b200 import ops
    w = H.QWeight(K, K, awq=awq, seed=K + M, name="gi").gpu(dev)
    x = torch.from_numpy(H.rng_for("gi-x", M).standard_normal((M, K)).astype(np.float16)).cuda()
    want = ops.matmul_affine(w, x)
    assert torch.equal(ops.matmul_affine(w, x, out=x), want)


@pytest.mark.parametrize("awq", [False, True])
@pytest.mark.parametrize("K,M", [(512, 16), (512, 130), (4096, 300)])
def test_rows_that_are_not_aligned(dev, K, M, awq):
    from ironmill_b200 import CudaSysError, ops
    w = H.QWeight(K, K, awq=awq, seed=K + M, name="gu").gpu(dev)
    x = torch.from_numpy(H.rng_for("gu-x", M).standard_normal((M, K)).astype(np.float16)).cuda()
    want = ops.matmul_affine(w, x)
    far = torch.empty(2, M * K + 8, dtype=torch.float16, device="cuda")
    xo, yo = far[0, 1:1 + M * K].view(M, K), far[1, 3:3 + M * K].view(M, K)
    xo.copy_(x)
    assert H.rel_err(ops.matmul_affine(w, xo, out=yo).cpu().numpy(), want.cpu().numpy()) <= TOL  # (K may be split for one and not the other)
    with pytest.raises(CudaSysError):
        ops.matmul_affine(w, xo, scratch=yo)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("K,M", [(1024, 7), (2048, 32), (1024, 48)])
def test_scratch_that_shares_memory(dev, K, M, bits):
    # without activation scales, tokens that can be read where they are stay there: a view at an offset into the scratch, and the result in the scratch
    from ironmill_b200 import ops
    w = H.QWeight(K, K, bits=bits, seed=K + M, name="gs").gpu(dev)
    x = torch.from_numpy(H.rng_for("gs-x", M).standard_normal((M, K)).astype(np.float16)).cuda()
    want = ops.matmul_affine(w, x).cpu().numpy()
    for at in (0, 8, 5 * K // 2, M * K - 8):  # from the same place to all but sixteen bytes apart
        buf = torch.zeros(2 * M * K, dtype=torch.float16, device="cuda")
        view = buf[at:at + M * K].view(M, K)
        view.copy_(x)
        assert H.rel_err(ops.matmul_affine(w, view, scratch=buf[:M * K]).cpu().numpy(), want) <= TOL, at
        assert torch.equal(view, x), at
        buf.zero_()
        out = ops.matmul_affine(w, x, out=buf[at:at + M * K].view(M, K), scratch=buf[:M * K])
        assert H.rel_err(out.cpu().numpy(), want) <= TOL, at


@pytest.mark.parametrize("N,K,M", [(19200, 1024, 24), (9600, 1024, 40), (256, 4096, 100)])
def test_two_streams(dev, N, K, M):
    # calls that keep nothing in the device handle: one beside another and beside a matvec, many row tiles and K slices of more than 64 tokens
    from ironmill_b200 import ops
    weights = [H.QWeight(N, K, seed=N + i, name="g2").gpu(dev) for i in range(2)]
    xs = [torch.from_numpy(H.rng_for("g2-x", i).standard_normal((M, K)).astype(np.float16)).cuda() for i in range(2)]
    want = [ops.matmul_affine(w, x) for w, x in zip(weights, xs)]
    vec = ops.matvec_affine(weights[0], xs[0][:2])
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got = [[], [], []]
    for _ in range(40):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got[i].append(ops.matmul_affine(weights[i], xs[i]) if i < 2 else ops.matvec_affine(weights[0], xs[0][:2]))
    torch.cuda.synchronize()
    for i, ref in enumerate(want + [vec]):
        assert all(torch.equal(y, ref) for y in got[i]), i


@pytest.mark.parametrize("awq", [False, True])
@pytest.mark.parametrize("K,M", [(1024, 5), (2048, 24), (1024, 48)])
def test_few_tokens_anywhere(dev, K, M, awq):
    # few tokens over a long sum: the result over the tokens, tokens and result at places that no vector reaches
    from ironmill_b200 import CudaSysError, ops
    w = H.QWeight(K, K, awq=awq, seed=K + M, name="gu").gpu(dev)
    x = torch.from_numpy(H.rng_for("gu-x", M).standard_normal((M, K)).astype(np.float16)).cuda()
    want = ops.matmul_affine(w, x)
    far = torch.empty(2, M * K + 8, dtype=torch.float16, device="cuda")
    xo, yo = far[0, 1:1 + M * K].view(M, K), far[1, 3:3 + M * K].view(M, K)
    xo.copy_(x)
    assert torch.equal(ops.matmul_affine(w, xo, out=yo), want)
    assert torch.equal(ops.matmul_affine(w, xo, out=xo), want)
    with pytest.raises(CudaSysError):
        ops.matmul_affine(w, yo, scratch=far[0, 1:1 + M * K].view(M, K))
    assert torch.equal(ops.matmul_affine(w, x, out=x), want)


def test_matches_the_matvec_kernel_rows(dev):
    # the same weight through the decode matvec (24-bit integer activations) and the GEMM: both within their tolerance of the oracle
    from ironmill_b200 import ops
    qw = H.QWeight(512, 1024, awq=True, seed=11, name="gm")
    w = qw.gpu(dev)
    x = torch.from_numpy(H.rng_for("gm-x").standard_normal((20, 1024)).astype(np.float16)).cuda()
    a = ops.matmul_affine(w, x).cpu().numpy().astype(np.float64)
    b = ops.matvec_affine(w, x).cpu().numpy().astype(np.float64)
    assert np.abs(a - b).max() / np.abs(b).max() <= 4e-3
