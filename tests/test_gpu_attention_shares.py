"""Decode attention of several contexts dealt out as equal shares of their tiles, against the same contexts cut by a split count that the caller gives."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests import helpers as H

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 2e-3  # fp16 operands, f32 sums in another order: the tolerance of these kernels against the oracle


# contexts long enough for shares and not; one and many, the most that are dealt out and one more; lengths of a tile and one more or less, one position, far apart (a share then spans several contexts, a context
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
