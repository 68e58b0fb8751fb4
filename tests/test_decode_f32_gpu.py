"""fp32 K/V on the TMA decode kernel against the CPU checker, 1e-5: group sizes below its eight head columns, both
head dims, slab edges (16 keys), whole-history units, chunks, shares and the cluster form."""
import numpy as np
import pytest

from tests.gpu_util import Case, check_case, from_device

pytestmark = pytest.mark.gpu


def make(orc, pkv, qh, kvh, hd, bs, ctx, seed):
    nb = sum((c + bs) // bs for c in ctx) + 9
    return Case(orc, "f32", qh, kvh, hd, bs, nb, ctx, [1] * len(ctx), seed=seed, pkv=pkv)


@pytest.mark.parametrize("qh,kvh", [(2, 2), (6, 2), (4, 1), (10, 2), (14, 2), (16, 2)])
@pytest.mark.parametrize("hd,bs", [(64, 16), (64, 64), (128, 16), (128, 32)])
def test_groups_and_slab_edges(pkv, orc, torch_cuda, qh, kvh, hd, bs):
    ctx = [0, 1, 14, 15, 16, 17, 31, 32, 47, 127, 128, 129, 300]
    case = make(orc, pkv, qh, kvh, hd, bs, ctx, seed=qh + hd)
    for mode in ("direct", "split", "device_plan"):
        check_case(case, pkv, torch_cuda, orc, mode)


@pytest.mark.parametrize("hd", [64, 128])
def test_shares(pkv, orc, torch_cuda, hd):
    """Enough keys that the plan is cut into one share per resident warp, at both head dims."""
    ctx = [int(x) for x in np.random.default_rng(2).integers(200, 9000, size=40)]
    case = make(orc, pkv, 8, 4, hd, 16, ctx, seed=3)
    for mode in ("host_plan", "device_plan"):
        check_case(case, pkv, torch_cuda, orc, mode)


@pytest.mark.parametrize("ctx", [[511] * 8, [333], [0, 2000, 15, 16, 17, 700], list(range(120, 160))])
def test_cluster_form(pkv, orc, torch_cuda, ctx):
    case = make(orc, pkv, 14, 2, 64, 16, ctx, seed=4)
    d = case.run_gpu(pkv, torch_cuda, "host_plan")
    before = pkv.lib().pkv_debug_cluster_launches()
    check_case(case, pkv, torch_cuda, orc, "host_plan")
    assert d["plan"].plan.cluster >= 2 and pkv.lib().pkv_debug_cluster_launches() == before + 1


def in_64_bits(case):
    out = np.empty((case.N, case.qh, case.hd))
    kc, vc = (x.copy().reshape(-1, case.kvh, case.hd).astype(np.float64) for x in (case.kc, case.vc))
    kc[case.idx.slots], vc[case.idx.slots] = (x.reshape(-1, case.kvh, case.hd) for x in (case.k, case.v))
    for t in range(case.N):
        pos = np.arange(case.idx.token_pos[t] + 1)
        table = case.idx.block_tables[case.idx.table_offset[case.idx.token_seq[t]]:]
        rows = table[pos // case.bs] * case.bs + pos % case.bs
        q = case.q[t].reshape(case.kvh, -1, case.hd).astype(np.float64)
        s = np.einsum("gid,kgd->gik", q, kc[rows]) * case.scale
        w = np.exp(s - s.max(-1, keepdims=True))
        out[t] = np.einsum("gik,kgd->gid", w / w.sum(-1, keepdims=True), vc[rows]).reshape(case.qh, case.hd)
    return out


@pytest.mark.parametrize("qh,kvh,hd,keys", [(4, 4, 64, 4000), (14, 2, 64, 8000), (8, 2, 128, 8000), (16, 2, 128, 3001)])
def test_long_histories_without_a_workspace(pkv, orc, torch_cuda, qh, kvh, hd, keys):
    """A whole history is summed by the four warps of a block.  A chain of n terms of random sign, each step rounded
    to 24 bits, ends up 2^-24 sqrt(n / 6) of the sum away; n = keys / 4, a fifth more allowed for the exponentials.
    (One chain of all the keys is twice that.)"""
    case = make(orc, pkv, qh, kvh, hd, 16, [keys - 1, keys - 20, keys - 333], seed=keys)
    check_case(case, pkv, torch_cuda, orc, "direct")
    got = from_device(torch_cuda, orc, case.run_gpu(pkv, torch_cuda, "direct")["out"], "f32")[1].reshape(case.N, qh, hd).astype(np.float64)
    want = in_64_bits(case)
    assert np.linalg.norm(got - want) <= 1.2 * 2.0 ** -24 * np.sqrt(keys / 24) * np.linalg.norm(want)


@pytest.mark.parametrize("keys,cluster", [(2048, False), (1000, True)])
def test_clusters_are_not_cut_below_the_rule(pkv, orc, torch_cuda, keys, cluster):
    """60 (token, kv head) pairs at 128 dims: four blocks each are offered and fp32 can hold two, which 2,048 keys are too
    many for (256 a warp); those take the ordinary form."""
    case = make(orc, pkv, 8, 4, 128, 16, [keys - 1] * 14 + [keys // 2], seed=6)
    before = pkv.lib().pkv_debug_cluster_launches()
    check_case(case, pkv, torch_cuda, orc, "host_plan")
    assert pkv.lib().pkv_debug_cluster_launches() == before + (1 if cluster else 0)
