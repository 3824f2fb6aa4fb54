"""Projections of few tokens (converted fragments on mma.sync) against the CPU oracle's matmul, and the forms of a model that chain them."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests import helpers as H
from tests.test_gpu_model import DictProvider, _cfg, synth_model

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 2e-3  # same fp16 operands, f32 accumulation in a different order, one fp16 rounding of the result


@pytest.fixture(scope="module")
def dev():
    from ironmill_b200 import ops
    return ops.Device(0)


# token counts around the eight tokens of an instruction and at the ends of both ranges; row counts that leave a row tile, a row block or eight
# rows incomplete; eight groups (one stage of a slice), an uneven number in slices, a long sum; more row tiles than CTAs
@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("N,K,M", [(16, 1024, 1), (120, 1024, 7), (200, 1408, 8), (1000, 1024, 9), (2056, 1152, 16), (136, 14336, 17), (6144, 1024, 24), (260, 2176, 25),
                                   (19208, 1024, 31), (24584, 1152, 12), (640, 4224, 32), (250, 1024, 33), (19000, 1280, 48), (512, 1024, 41)])
def test_few_tokens(dev, N, K, M, bits):
    from ironmill_b200 import ops
    qw = H.QWeight(N, K, bits=bits, awq=M % 2 == 0, seed=N + M + bits, name="gr")
    qw.zps = qw.zps.copy()
    qw.zps[3::397] += 0.25  # zero points that are no integer: the f32 path
    qw.zps[5::911] = -700.0  # and one past the range of the packed one
    qw.zps_f16 = orc.f32_to_f16(qw.zps)
    w = qw.gpu(dev)
    x = (H.rng_for("gr-x", M).standard_normal((M, K))).astype(np.float16)
    ref = orc.matmul_affine(qw.packed, qw.scales_f16, qw.zps_f16, x, N, K, 128, bits, awq=qw.awq, threads=8)
    for _ in range(2):  # the counters of cut tiles are back at zero after a launch
        y = ops.matmul_affine(w, torch.from_numpy(x).cuda()).cpu().numpy()
        assert H.rel_err(y, ref) <= TOL, (N, K, M)


# The same with the rows of far zero points, whose results are a hundred times the others', compared apart: an error of the size of an ordinary result
# shows in neither otherwise.
@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("N,K,M", [(16, 1024, 1), (200, 1408, 8), (1000, 1024, 9), (136, 14336, 17), (260, 2176, 25), (19208, 1024, 31), (640, 4224, 32), (250, 1024, 33), (19000, 1280, 48)])
def test_few_tokens_by_rows_of_like_size(dev, N, K, M, bits):
    from ironmill_b200 import ops
    qw = H.QWeight(N, K, bits=bits, awq=M % 2 == 0, seed=N + M + bits, name="gr")
    qw.zps = qw.zps.copy()
    qw.zps[3::397] += 0.25
    qw.zps[5::911] = -700.0
    qw.zps_f16 = orc.f32_to_f16(qw.zps)
    w = qw.gpu(dev)
    x = (H.rng_for("gr-x", M).standard_normal((M, K))).astype(np.float16)
    ref = orc.matmul_affine(qw.packed, qw.scales_f16, qw.zps_f16, x, N, K, 128, bits, awq=qw.awq, threads=8)
    far = np.zeros(N, dtype=bool)
    far[np.nonzero(np.abs(qw.zps.reshape(N, -1)) > 500)[0]] = True
    assert far.any() and not far.all()
    y = ops.matmul_affine(w, torch.from_numpy(x).cuda()).cpu().numpy()
    for part in (far, ~far):
        assert H.rel_err(y[:, part], ref[:, part]) <= TOL, (N, K, M)


@pytest.mark.parametrize("N,K,M", [(512, 2048, 65), (384, 1792, 128), (260, 14336, 100), (6144, 1024, 97)])
def test_one_token_tile_over_slices_of_k(dev, N, K, M):
    # the tcgen05 kernel's full token tile with K cut along the grid: ragged rows, an uneven last slice, both ends of the token range
    from ironmill_b200 import ops
    qw = H.QWeight(N, K, awq=True, seed=N + M, name="gs")
    x = (H.rng_for("gs-x", M).standard_normal((M, K))).astype(np.float16)
    y = ops.matmul_affine(qw.gpu(dev), torch.from_numpy(x).cuda()).cpu().numpy()
    ref = orc.matmul_affine(qw.packed, qw.scales_f16, qw.zps_f16, x, N, K, 128, 4, awq=qw.awq, threads=8)
    assert H.rel_err(y, ref) <= TOL, (N, K, M)


@pytest.mark.parametrize("chunk", [9, 24, 33])
def test_prompt_in_short_portions(chunk):
    """Portions of few tokens (packed norms, joint gate and up, packed activation) against the whole prompt at once (the kernels of many tokens):
    the same operands and rounding points, sums in another order, an fp16 cache.  Each of the layer's seven roundings to fp16 may fall the other way,
    2^-11 of a value each, two layers deep: sqrt(14) 2^-11 = 1.8e-3 of the logits' norm, doubled."""
    from ironmill_b200.engine import CudaConfig, CudaInference
    cfg = _cfg("llama", 2, 1024, 1152, 8, 4, 500, 1e6, 1e-6)
    tensors = synth_model(cfg, seed=31, gamma_jitter=0.2)
    tokens = H.rng_for("rows-prompt").integers(0, 500, 99).astype(np.uint32)
    out = []
    for c in (99, chunk):
        conf = CudaConfig(max_seq_len=128, max_batch=1, prefill_chunk_size=c)
        conf.without_turboquant()
        eng = CudaInference(conf)
        eng.load_weights(DictProvider(cfg, tensors))
        out.append(eng.prefill(tokens).astype(np.float64))
    assert np.linalg.norm(out[1] - out[0]) / np.linalg.norm(out[0]) <= 3.6e-3


@pytest.mark.parametrize("bits,chunk", [(4, 40), (8, 20)])
def test_prompt_whose_down_projection_is_another_kernel(bits, chunk):
    """Gate and up joint over packed tokens, the activation left unpacked for a down projection whose slices of K would be too long for clusters (8 row tiles
    of 14336 columns); against the prompt at once, the bound of the test above for one layer."""
    from ironmill_b200.engine import CudaConfig, CudaInference
    cfg = _cfg("llama", 1, 1024, 14336, 8, 4, 200, 1e6, 1e-6)
    tensors = synth_model(cfg, seed=33, awq=True, bits=bits)
    tokens = H.rng_for("rows-down").integers(0, 200, 3 * chunk).astype(np.uint32)
    out = []
    for c in (3 * chunk, chunk):
        conf = CudaConfig(max_seq_len=128, max_batch=1, prefill_chunk_size=c)
        conf.without_turboquant()
        eng = CudaInference(conf)
        eng.load_weights(DictProvider(cfg, tensors))
        out.append(eng.prefill(tokens).astype(np.float64))
    assert np.linalg.norm(out[1] - out[0]) / np.linalg.norm(out[0]) <= 3.6e-3


@pytest.mark.parametrize("bits,batch,chunk", [(4, 3, 24), (8, 9, 13), (4, 15, 48)])
def test_row_tiles_cut_by_shares(bits, batch, chunk):
    """Gate and up of more row tiles than SMs over a sum long enough for equal shares: tiles cut by CTA boundaries, launch after launch (the counters are back
    at zero).  A prompt in portions against the prompt at once, then steps over byte planes against the oracle model of the first sequences."""
    from ironmill_b200.engine import CudaConfig, CudaInference
    from tests.oracle_model import OracleModel
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    H_, tiles = 2048, sms + 4
    ff = tiles * 64 // 128 * 128  # a joint tile: 64 rows of each
    assert ff // 64 > sms and 2 * (H_ // 128) > (ff // 64) * (H_ // 128) / sms + 13
    cfg = _cfg("llama", 1, H_, ff, 8, 4, 200, 1e6, 1e-6)
    tensors = synth_model(cfg, seed=45, awq=True, bits=bits)
    tqc = orc.TqConstants(128, 8, seed=4)
    rng = H.rng_for("cut")
    prompt = rng.integers(0, 200, 2 * chunk).astype(np.uint32)
    prompts = [rng.integers(0, 200, 2 + i % 3).astype(np.uint32) for i in range(batch)]
    out = []
    for c in (2 * chunk, chunk):
        conf = CudaConfig(max_seq_len=128, max_batch=1, prefill_chunk_size=c)
        conf.without_turboquant()
        eng = CudaInference(conf)
        eng.load_weights(DictProvider(cfg, tensors))
        out.append(eng.prefill(prompt).astype(np.float64))
    assert np.linalg.norm(out[1] - out[0]) / np.linalg.norm(out[0]) <= 3.6e-3  # as test_prompt_in_short_portions
    eng = CudaInference(CudaConfig(max_seq_len=128, max_batch=batch, n_bits=8))
    eng.load_weights(DictProvider(cfg, tensors), tq_signs=tqc.signs, tq_qjl=tqc.qjl)
    ids = [eng.add_sequence(p) for p in prompts]
    refs = [OracleModel(cfg, tensors, tqc, 128) for _ in prompts[:2]]
    for ref, p in zip(refs, prompts):
        ref.forward(p)
    for _ in range(3):
        fed = rng.integers(0, 200, batch)
        got = eng.batch_decode_step(dict(zip(ids, fed.tolist())))
        for i, ref in enumerate(refs):
            assert float(np.abs(got[i][1] - ref.forward([int(fed[i])])).max()) <= 5e-2, (bits, batch, i)


@pytest.mark.parametrize("bits,awq,batch", [(4, True, 1), (4, True, 2), (4, False, 3), (8, True, 5), (4, True, 9), (8, False, 15)])
def test_decode_batches_over_planes(bits, awq, batch):
    """Steps of a few sequences (planes written by the norms, Q | K | V and gate | up joint) against the oracle model of the first ones, at the gate of decode
    logits: row counts around the two rows of an instruction, both code widths and their rounding points."""
    from ironmill_b200.engine import CudaConfig, CudaInference
    from tests.oracle_model import OracleModel
    cfg = _cfg("llama", 2, 1024, 1152, 8, 4, 300, 1e6, 1e-6)
    tensors = synth_model(cfg, seed=41, awq=awq, gamma_jitter=0.2, bits=bits)
    tqc = orc.TqConstants(128, 8, seed=4)
    eng = CudaInference(CudaConfig(max_seq_len=64, max_batch=max(batch, 2), n_bits=8))
    eng.load_weights(DictProvider(cfg, tensors), tq_signs=tqc.signs, tq_qjl=tqc.qjl)
    rng = H.rng_for("planes")
    prompts = [rng.integers(0, 300, 3 + i % 5).astype(np.uint32) for i in range(batch)]
    ids = [eng.add_sequence(p) for p in prompts]
    refs = [OracleModel(cfg, tensors, tqc, 64) for _ in prompts[:3]]
    for ref, p in zip(refs, prompts):
        ref.forward(p)
    for _ in range(3):
        fed = rng.integers(0, 300, batch)
        got = eng.batch_decode_step(dict(zip(ids, fed.tolist())))
        for i, ref in enumerate(refs):
            want = ref.forward([int(fed[i])])
            assert float(np.abs(got[i][1] - want).max()) <= 5e-2, (bits, batch, i)
