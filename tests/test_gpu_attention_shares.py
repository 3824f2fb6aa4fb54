"""Decode attention of several contexts dealt out as equal shares of their tiles, against the same contexts cut by a split count that the caller gives."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests import helpers as H

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 2e-3  # fp16 operands, f32 sums in another order: the tolerance of these kernels against the oracle


# contexts long enough for shares and not; several and many, the most that are dealt out and one more; lengths of a tile and one more or less, one position, far apart (a share then spans several contexts, a context
# several shares); one query head per KV head and four; both cache widths
@pytest.mark.parametrize("bits,nh", [(8, 8), (4, 8), (8, 2)])
@pytest.mark.parametrize("lengths", [(3000,), (70000,), (1, 60000, 33, 32, 31, 18000), tuple(1 + 97 * i % 3500 for i in range(64)), tuple(1 + 61 * i % 400 for i in range(65))])
def test_shares_of_unequal_contexts(bits, nh, lengths):
    from ironmill_b200 import ops
    dev, nkv, n, ctx = ops.Device(0), 2, len(lengths), max(lengths) + 5
    tqc = orc.TqConstants(128, bits, seed=6)
    tq = ops.TurboQuant(dev, 128, bits, tqc.signs, tqc.qjl)
    rng = H.rng_for("shares", n + bits)
    cache = {}
    for part in "kv":
        rows = torch.from_numpy(rng.standard_normal((n * ctx, nkv, 128)).astype(np.float16)).cuda()
        cache[part] = torch.zeros((n, nkv, ctx, 128 * bits // 8), dtype=torch.uint8, device="cuda")
        cache[part + "s"] = torch.zeros((n, nkv, ctx), device="cuda")
        cache[part + "r"] = torch.zeros((n, nkv, ctx), device="cuda") if part == "k" else None
        tq.encode(rows, part == "k", cache[part], cache[part + "s"], cache[part + "r"], nkv, ctx, 0, nseq=n)
    q = torch.from_numpy(rng.standard_normal((n, nh, 128)).astype(np.float16)).cuda()
    pos = torch.tensor([x - 1 for x in lengths], dtype=torch.int32, device="cuda")

    def run(splits):
        return tq.attention(q, cache["k"], cache["v"], cache["ks"], cache["vs"], cache["kr"], 128 ** -0.5, nh, nkv, ctx, 0, nseq=n, pos_dev=pos, num_splits=splits).float().cpu().numpy()

    want = run(3)
    for _ in range(2):
        got = run(0)
        for i in range(n):
            assert H.rel_err(got[i], want[i]) <= TOL, lengths[i]


def _caches(tq, n, nkv, ctx, bits, seed):
    rng = torch.Generator(device="cuda").manual_seed(seed)
    cache = {}
    for part in "kv":
        cache[part] = torch.zeros((n, nkv, ctx, 128 * bits // 8), dtype=torch.uint8, device="cuda")
        cache[part + "s"] = torch.zeros((n, nkv, ctx), device="cuda")
        cache[part + "r"] = torch.zeros((n, nkv, ctx), device="cuda") if part == "k" else None
        tq.encode(torch.randn((n * ctx, nkv, 128), generator=rng, device="cuda").half(), part == "k", cache[part], cache[part + "s"], cache[part + "r"], nkv, ctx, 0, nseq=n)
    return cache


def _long(sms, contexts):
    """Positions with which so many contexts can just be dealt out: 16 tiles of 32 for two CTAs per SM."""
    return -(-2 * sms * 16 // contexts) * 32


# lengths as parts of the shortest cache with which a launch may take shares: one context (above, at and below 8 tiles a CTA), one that sees nothing, one far
# longer than the others (parts after all), the most contexts that have a CTA each and one token more, several tokens of a sequence
@pytest.mark.parametrize("bits,gq,nkv,T,lengths", [
    (8, 4, 2, 1, (1.0,)), (4, 2, 8, 1, (0.52,)), (8, 1, 2, 1, (0.4,)), (8, 2, 4, 1, (1.0, 0.0, 0.7, 0.01)), (8, 4, 8, 1, (1.0,) + (0.02,) * 15), (4, 4, 2, 1, (0.9, 0.3, 1.0)),
    (8, 2, 8, 1, tuple(0.5 + i % 7 / 14 for i in range(37))), (8, 2, 8, 1, tuple(0.5 + i % 7 / 14 for i in range(38))), (8, 2, 8, 3, (1.0, 0.4, 0.8, 0.6)), (4, 1, 8, 16, (1.0, 0.7))])
def test_shares_over_what_launches_have(bits, gq, nkv, T, lengths):
    from ironmill_b200 import ops
    dev, n, nh = ops.Device(0), len(lengths), gq * nkv
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ctx = _long(sms, n * T * nkv) + 32
    tqc = orc.TqConstants(128, bits, seed=6)
    tq = ops.TurboQuant(dev, 128, bits, tqc.signs, tqc.qjl)
    c = _caches(tq, n, nkv, ctx, bits, n + T)
    q = torch.randn((n, T, nh, 128), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").half()
    pos = torch.tensor([max(int(x * (ctx - T)) - 1, -T) for x in lengths], dtype=torch.int32, device="cuda")

    def run(splits):
        return tq.attention(q, c["k"], c["v"], c["ks"], c["vs"], c["kr"], 128 ** -0.5, nh, nkv, ctx, 0, nseq=n, pos_dev=pos, num_splits=splits).float().cpu().numpy()

    want, got = run(3), run(0)
    assert np.isfinite(got).all()
    for i in range(n):
        for t in range(T):
            if lengths[i] == 0.0:
                assert not got[i, t].any() and not want[i, t].any()
            else:
                assert H.rel_err(got[i, t], want[i, t]) <= TOL, (i, t)


def test_steps_over_cache_slots():
    """Batched steps of an engine whose contexts are dealt out (captured, slots that are not the first ones) against steps of fewer sequences, which are not:
    sums in another order; the bound of test_gpu_gemm_rows.test_prompt_in_short_portions."""
    from ironmill_b200.engine import CudaConfig, CudaInference
    from tests.test_gpu_model import DictProvider, _cfg, synth_model
    cfg = _cfg("llama", 2, 1024, 1152, 8, 8, 300, 1e6, 1e-6)
    tensors = synth_model(cfg, seed=12, gamma_jitter=0.2)
    tqc = orc.TqConstants(128, 8, seed=4)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ctx = _long(sms, 7 * 8) + 64
    rng = H.rng_for("slots")
    prompts = [rng.integers(0, 300, int(ctx * (0.5 + 0.06 * i))).astype(np.uint32) for i in range(8)]
    fed = rng.integers(0, 300, (3, 8))
    engines = []
    for _ in range(2):
        eng = CudaInference(CudaConfig(max_seq_len=ctx, max_batch=8, n_bits=8))
        eng.load_weights(DictProvider(cfg, tensors), tq_signs=tqc.signs, tq_qjl=tqc.qjl)
        engines.append((eng, [eng.add_sequence(p) for p in prompts]))
    for step in fed:
        out = []
        for (eng, ids), groups in zip(engines, ([range(1, 8)], [range(1, 4), range(4, 8)])):
            got = {}
            for g in groups:
                got.update(dict(eng.batch_decode_step({ids[i]: int(step[i]) for i in g})))
            out.append([got[ids[i]].astype(np.float64) for i in range(1, 8)])
        for a, b in zip(*out):
            assert np.linalg.norm(a - b) / np.linalg.norm(b) <= 3.6e-3
