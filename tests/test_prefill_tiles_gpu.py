"""Query tiles that hold several heads of a group: every packing the launcher chooses, chunk lengths around its
tile, and the order the tiles are handed out in (one, a few dozen, and more sequences than are ranked)."""
import numpy as np
import pytest

from tests.gpu_util import TOL, from_device, rel_errors
from tests.test_prefill_gpu import make_case, run_prefill

pytestmark = pytest.mark.gpu


def check(pkv, orc, torch, qh, kvh, ctx, new, seed, dtype="bf16"):
    case = make_case(orc, pkv, dtype, qh, kvh, 16, ctx, new, seed)
    _, _, want = case.expected(orc, threads=8)
    d = run_prefill(pkv, torch, case)
    _, got = from_device(torch, orc, d["out"], dtype)
    assert np.isfinite(got).all()
    e_ref, e_row = rel_errors(got.reshape(-1, 64), want.reshape(-1, 64))
    assert e_ref <= TOL[dtype] and e_row <= TOL[dtype], (e_ref, e_row)


@pytest.mark.parametrize("group", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 13, 16, 20, 28])
def test_every_packing(pkv, orc, torch_cuda, group):
    """Tiles of 128 / heads tokens: 8 (16 heads) to 128 (one head; also a group of 13, which would waste rows)."""
    pack = max(p for p in range(1, 17) if group % p == 0 and (p == 1 or 128 // p * p >= 120))
    tt = 128 // pack
    check(pkv, orc, torch_cuda, 2 * group, 2, [0, 5, 64, 190, 0], [tt - 1, tt, tt + 1, 2 * tt + 3, 1], seed=group)


@pytest.mark.parametrize("n_seqs", [1, 31, 33, 70, 257])
def test_many_sequences(pkv, orc, torch_cuda, n_seqs):
    rng = np.random.default_rng(n_seqs)
    ctx = [int(x) for x in rng.integers(0, 300, size=n_seqs)]
    new = [int(x) for x in rng.integers(1, 60, size=n_seqs)]
    check(pkv, orc, torch_cuda, 14, 2, ctx, new, seed=5, dtype="f16")


def test_equal_lengths(pkv, orc, torch_cuda):
    """Every tile of a rank has the same length as its neighbours: one bucket, many ties."""
    check(pkv, orc, torch_cuda, 8, 1, [64] * 24, [48] * 24, seed=6)


@pytest.mark.parametrize("qh,kvh", [(14, 2), (8, 1), (26, 2), (32, 4)])
@pytest.mark.parametrize("ctx,new", [
    ([3000], [1]),                       # one tile, all eight blocks of a cluster on it
    ([0], [250]),                        # parts of the keys that early rows do not see
    ([5000, 64, 127], [33, 17, 60]),     # long and short items in one launch
    ([700, 900, 1100], [70, 71, 140]),   # two and four blocks per item
    ([63], [1]), ([64], [2]),            # around one key tile: nothing to share
])
def test_few_items_share_their_keys(pkv, orc, torch_cuda, qh, kvh, ctx, new):
    check(pkv, orc, torch_cuda, qh, kvh, ctx, new, seed=7)


def test_split_launch_replays_from_a_graph(pkv, orc, torch_cuda):
    torch = torch_cuda
    case = make_case(orc, pkv, "bf16", 14, 2, 16, [2000, 900], [40, 25], seed=8)
    d = run_prefill(pkv, torch, case)
    want = d["out"].clone()
    i32 = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()
    args = (i32([0, 40]), i32([40, 25]), i32([2000, 900]))
    out = torch.zeros_like(want)
    call = lambda: pkv.launch_attention_prefill(d["q"], d["kc"], d["vc"], d["block_tables"], d["table_offset"], *args, out,
                                                case.N, 2, 40, 14, 2, 64, 16, case.nb, case.scale)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for _ in range(5):
            call()
    for _ in range(3):
        out.zero_()
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and pkv.debug_device_flags() == 0


@pytest.mark.parametrize("qh,kvh", [(14, 2), (3, 3)])
@pytest.mark.parametrize("n_seqs,longest", [(30, 1), (32, 700), (64, 250), (96, 130), (255, 90), (256, 300), (257, 40)])
def test_lists_of_tiles(pkv, orc, torch_cuda, qh, kvh, n_seqs, longest):
    """One slot per block, a list in the sequences' order, and one ordered by length, over 32, 64, ... sequences:
    every row of every chunk is written, whatever the lengths and whichever sequences bring nothing."""
    rng = np.random.default_rng(n_seqs)
    ctx = [int(x) for x in rng.integers(0, longest, size=n_seqs)]
    new = [int(x) for x in rng.integers(1, 1 + min(longest, 70), size=n_seqs)]
    new[n_seqs // 2] = min(longest, 200)
    check(pkv, orc, torch_cuda, qh, kvh, ctx, new, seed=n_seqs, dtype="f16")


@pytest.mark.parametrize("ctx,new", [([0, 300, 0, 40], [60, 60, 60, 60]), ([0, 0, 0], [100, 90, 100]), ([3, 0, 900, 0, 64], [1, 200, 17, 3, 130])])
def test_few_items_of_uneven_sequences(pkv, orc, torch_cuda, ctx, new):
    """Clusters for more slots than items: the tiles come from the list."""
    for qh, kvh in ((14, 2), (8, 1), (2, 2)):
        check(pkv, orc, torch_cuda, qh, kvh, ctx, new, seed=10)


def test_a_generous_longest_chunk(pkv, orc, torch_cuda):
    """max_q_len is an upper bound: 2^30 makes 2^29 slots, which eight blocks each would count past 32 bits."""
    torch = torch_cuda
    ctx, new = [0, 3, 64, 700, 0, 90, 5, 17], [1, 5, 2, 1, 3, 1, 4, 1]
    case = make_case(orc, pkv, "bf16", 8, 1, 16, ctx, new, seed=11)
    _, _, want = case.expected(orc, threads=4)
    d = run_prefill(pkv, torch, case)
    i32 = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()
    d["out"].fill_(float("nan"))
    pkv.launch_attention_prefill(d["q"], d["kc"], d["vc"], d["block_tables"], d["table_offset"], i32(np.cumsum(new) - new), i32(new), i32(ctx),
                                 d["out"], case.N, len(new), 1 << 30, 8, 1, 64, 16, case.nb, case.scale)
    torch.cuda.synchronize()
    _, got = from_device(torch, orc, d["out"], "bf16")
    e_ref, e_row = rel_errors(got.reshape(-1, 64), want.reshape(-1, 64))
    assert e_ref <= TOL["bf16"] and e_row <= TOL["bf16"] and pkv.debug_device_flags() == 0
