"""The split-K work list (csrc/decode_plan.hpp): every token's keys exactly once, partial slots distinct, shares
that cover the items in order and hold about the same number of keys.  The host planner is read back from
its image; the device planner has to produce the same integers."""
import ctypes as C

import numpy as np
import pytest

SLAB, MIN_SHARE = 32, 128


def align256(n):
    return (n + 255) // 256 * 256


def host_image(pkv, pos, qh, kvh, hd, ws_bytes=None):
    L = pkv.lib()
    pos = np.ascontiguousarray(pos, dtype=np.int32)
    nstage = L.pkv_decode_plan_staging_bytes(pos.size, kvh)
    staging = np.zeros(nstage, dtype=np.uint8)
    plan, image = pkv._lib.DecodePlan(), C.c_size_t(0)
    ws = ws_bytes or L.pkv_decode_workspace_bytes(pos.size, qh, kvh, hd)
    st = L.pkv_decode_plan_host_image(pos.ctypes.data, pos.size, qh, kvh, hd, staging.ctypes.data, nstage, ws, C.byref(plan), C.byref(image))
    assert st == 0, L.pkv_last_error()
    return staging[:image.value], plan


def read(image, n, kvh):
    """(header, splits, items, first item of every share) of a plan image."""
    words = image.view(np.int32)
    header = words[:8]
    o = 256
    splits = words[o // 4:o // 4 + 2 * n].reshape(n, 2)
    o = align256(align256(o + 8 * n) + 4 * n * kvh)
    items = words[o // 4:o // 4 + 4 * header[1]].reshape(-1, 4)
    first = words[o // 4 + 4 * header[1]:][:header[6] + 1] if header[6] else None
    return header, splits, items, first


def check(image, pos, kvh):
    n = len(pos)
    header, splits, items, first = read(image, n, kvh)
    assert header[3] == n and header[5] == kvh
    seen = np.zeros(header[4], dtype=int)
    for t in range(n):
        mine = items[items[:, 0] == t]
        assert len(mine) == splits[t, 1]
        mine = mine[np.argsort(mine[:, 1])]
        at = 0
        for s, (_, b, ln, part) in enumerate(mine):
            assert b == at and ln > 0 and (b % SLAB == 0)
            assert part == (splits[t, 0] + s if len(mine) > 1 else -1)
            if part >= 0:
                seen[part] += 1
            at += ln
        assert at == pos[t] + 1
    assert (seen == 1).all()
    if first is not None:
        per, n_shares = header[2], header[6]
        assert first[0] == 0 and first[-1] == header[1] and (np.diff(first) >= 0).all() and (np.diff(first)[:-1] > 0).all()
        padded = [sum(-(-x // SLAB) * SLAB for x in items[first[s]:first[s + 1], 2]) for s in range(n_shares)]
        assert max(padded) <= per + 2 * SLAB and min(padded[:-1], default=per) >= per - 2 * SLAB
        assert items[:, 2].min() > 0 and all(x > SLAB for t in range(n) if splits[t, 1] > 1 for x in items[items[:, 0] == t, 2])
    return header


STEPS = {
    "one": [0], "one long": [70000], "slab edges": [30, 31, 32, 33, 63, 64, 65, 95, 96, 127, 128] * 40,
    "small": [5, 300, 17, 129, 1500], "none long": [127, 3, 90, 64, 65, 127], "fine or not": [128] * 60, "equal": [4095] * 256, "short": [99] * 1500, "single keys": [0] * 2500,
    "ragged": np.random.default_rng(3).integers(0, 8192, size=256), "last token of one slab": [127] * 3551 + [31],
}


@pytest.mark.parametrize("kvh", [1, 2, 4, 8])
@pytest.mark.parametrize("name", sorted(STEPS))
def test_host_plan_covers_every_key_once(pkv, name, kvh):
    pos = np.asarray(STEPS[name], dtype=np.int32)
    for hd in (64, 128):
        check(host_image(pkv, pos, 4 * kvh, kvh, hd)[0], pos, kvh)


@pytest.mark.parametrize("extra", [0, 1, 2, 3, 7, 40, 200])
def test_small_workspaces_take_fewer_shares(pkv, extra):
    """The partials (2 * extra slots) and the share table stay inside what the workspace was sized for."""
    pos, qh, kvh, hd = np.random.default_rng(4).integers(0, 4096, size=60).astype(np.int32), 8, 2, 64
    n = pos.size
    off_items = align256(align256(256 + 8 * n) + 4 * n * kvh)
    ml = align256(off_items + 16 * (n + extra))
    total = align256(align256(ml + 8 * 2 * extra * qh) + 4 * 2 * extra * qh * hd)
    image, plan = host_image(pkv, pos, qh, kvh, hd, total)
    header = check(image, pos, kvh)
    assert header[4] <= 2 * extra and image.size <= ml


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(STEPS))
def test_device_plan_is_the_host_plan(pkv, torch_cuda, name):
    """Same cuts, slots and shares, around the 1,024 tokens one pass of the planner block takes (chunked steps
    list the items in another order, and may have chunks half as long)."""
    torch = torch_cuda
    pos = np.asarray(STEPS[name], dtype=np.int32)
    for n in sorted({pos.size, min(pos.size, 1024), min(pos.size, 1025)}):
        p = np.ascontiguousarray(pos[:n])
        plan = pkv.DecodePlan(n, 32, 4, 64)
        plan.workspace.random_(0, 255)
        plan.build_device(torch.from_numpy(p).cuda())
        torch.cuda.synchronize()
        got = read(plan.workspace.cpu().numpy(), n, 4)
        image, _ = host_image(pkv, p, 32, 4, 64)
        want = read(image, n, 4)
        check(plan.workspace.cpu().numpy(), p, 4)
        if want[3] is None and got[0][2] == MIN_SHARE // 2:
            assert want[0][2] == MIN_SHARE and p.max() >= MIN_SHARE and got[3] is None
            continue
        assert got[0].tolist() == want[0].tolist() and (got[1][:, 1] == want[1][:, 1]).all()
        key = lambda items: sorted(map(tuple, items.tolist()))
        assert key(got[2]) == key(want[2])
        if want[3] is not None:
            assert (got[3] == want[3]).all() and (got[2] == want[2]).all()


def ragged(n, lo, hi, seed=5):
    return np.random.default_rng(seed).integers(lo, hi, size=n).astype(np.int32)


@pytest.mark.parametrize("qh,kvh,hd", [(32, 1, 64), (16, 4, 96), (8, 2, 256), (40, 2, 128)])
def test_kernels_that_give_an_item_a_block_get_chunks(pkv, qh, kvh, hd):
    """Head dims other than 64 and 128 and groups above 16: chunks, full ones first, however many keys there are."""
    pos = ragged(200, 100, 2000)
    header, _, items, first = read(host_image(pkv, pos, qh, kvh, hd)[0], pos.size, kvh)
    assert first is None and header[2] in (128, 256, 512) and (np.diff(items[:, 2]) <= 0).all()
    check(host_image(pkv, pos, qh, kvh, hd)[0], pos, kvh)
    assert read(host_image(pkv, pos, 32, 4, 64)[0], pos.size, 4)[3] is not None


def test_steps_of_many_short_tokens_are_not_cut(pkv):
    """Whole tokens fill the GPU: no partials, and so no merge launch; a few longer ones are cut as before."""
    for kvh, most in ((2, 199), (2, 100), (4, 199), (8, 199)):
        pos = ragged(1000, 20, most)
        image, plan = host_image(pkv, pos, 4 * kvh, kvh, 64)
        header = check(image, pos, kvh)
        assert header[4] == 0 and plan.reserved == 0 and header[6] == 0
    assert check(host_image(pkv, ragged(60, 20, 199), 16, 4, 64)[0], ragged(60, 20, 199), 4)[4] > 0


def test_shares_are_for_tokens_longer_than_a_share(pkv):
    """Up to 192 keys a share: chunks where the tokens are mostly shorter than two shares."""
    short, long = ragged(600, 60, 440), np.full(8, 2999, np.int32)
    assert check(host_image(pkv, short, 14, 2, 64)[0], short, 2)[6] == 0
    assert check(host_image(pkv, short, 32, 4, 64)[0], short, 4)[6] > 0        # 370 keys a share
    assert check(host_image(pkv, long, 32, 8, 128)[0], long, 8)[6] > 0         # 162


@pytest.mark.gpu
@pytest.mark.parametrize("pos,chunk", [([2047], 64), ([2048], 128), ([7999], 128), ([2999] * 8, 128), ([900, 100, 400, 300, 250, 128], 64),
                                       ([127] * 30, 128)])
def test_half_chunks_are_for_short_histories(pkv, torch_cuda, pos, chunk):
    """Chunks of 64 keys: something to merge (a token above 128 keys) and no token of more than 32 of them."""
    plan = pkv.DecodePlan(len(pos), 14, 2, 64).build_device(torch_cuda.tensor(pos, dtype=torch_cuda.int32, device="cuda"))
    torch_cuda.cuda.synchronize()
    image = plan.workspace.cpu().numpy()
    check(image, pos, 2)
    assert read(image, len(pos), 2)[0][2] == chunk


@pytest.mark.parametrize("kvh,hd,seqs,keys,size,least", [(2, 64, 50, 4096, 4, 4), (2, 64, 50, 2049, 4, 3), (4, 128, 15, 2048, 4, 4), (4, 128, 15, 700, 4, 2),
                                                         (2, 64, 1, 300, 8, 1)])
def test_smallest_cluster_the_rule_allows(pkv, kvh, hd, seqs, keys, size, least):
    """256 keys a warp (128 at 128 dims), four warps a block: what a launch may shrink the offered clusters to."""
    plan = host_image(pkv, np.full(seqs, keys - 1, np.int32), 2 * kvh, kvh, hd)[1]
    assert (plan.cluster if hd == 64 else plan.cluster_wide) == size and plan.cluster_least == least
