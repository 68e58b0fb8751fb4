"""Mixed steps around the size up to which the kernels plan for themselves (704 tokens, 256 runs): the same step
through the planner launch and without it, against the CPU checker."""
import numpy as np
import pytest

from tests.gpu_util import Case, TOL, from_device, rel_errors

pytestmark = pytest.mark.gpu


def run(pkv, orc, torch, dtype, qh, kvh, ctx, new, seed, min_run=0):
    nb = sum((c + n + 15) // 16 for c, n in zip(ctx, new)) + 9
    case = Case(orc, dtype, qh, kvh, 64, 16, nb, ctx, new, seed=seed, pkv=pkv)
    _, _, want = case.expected(orc, threads=8)
    d = case.upload(torch)
    pkv.launch_store_kv(d["k"], d["v"], d["slots"], d["kc"], d["vc"], case.N, kvh * 64)
    ws = torch.empty(pkv.mixed_workspace_bytes(case.N, qh, kvh, 64), dtype=torch.uint8, device="cuda").random_(0, 255)
    for _ in range(3):                                   # back to back: the launches of one step overlap those of the next
        d["out"].fill_(float("nan"))
        for _ in range(4):
            pkv.launch_attention_mixed(d["q"], d["kc"], d["vc"], d["block_tables"], d["table_offset"], d["token_seq"], d["token_pos"],
                                       d["out"], case.N, qh, kvh, 64, 16, case.scale, ws, num_blocks=nb, min_run=min_run)
    torch.cuda.synchronize()
    _, got = from_device(torch, orc, d["out"], dtype)
    e_ref, e_row = rel_errors(got.reshape(-1, 64), want.reshape(-1, 64))
    assert e_ref <= TOL[dtype] and e_row <= TOL[dtype] and pkv.debug_device_flags() == 0, (e_ref, e_row)


@pytest.mark.parametrize("total", [16, 128, 129, 703, 704, 705])
def test_token_counts(pkv, orc, torch_cuda, total):
    """Two prompt chunks (when they fit), the rest decode tokens of all lengths."""
    rng = np.random.default_rng(total)
    chunks = [150, 33] if total > 200 else []
    n = total - sum(chunks)
    run(pkv, orc, torch_cuda, "f16", 14, 2, [40, 700] [:len(chunks)] + [int(x) for x in rng.integers(0, 400, size=n)], chunks + [1] * n, seed=total)


@pytest.mark.parametrize("qh,kvh", [(4, 4), (32, 2), (8, 1)])
def test_shares_and_groups(pkv, orc, torch_cuda, qh, kvh):
    """Histories long enough for equal shares per warp, chunks between and behind the decode tokens."""
    rng = np.random.default_rng(7)
    ctx = [int(x) for x in rng.integers(1500, 6000, size=70)]
    new = [1] * 70
    for at, n in ((0, 20), (30, 64), (69, 17)):
        new[at] = n
    run(pkv, orc, torch_cuda, "bf16", qh, kvh, ctx, new, seed=8)


@pytest.mark.parametrize("min_run", [1, 2, 3, 1000])
def test_run_lengths(pkv, orc, torch_cuda, min_run):
    run(pkv, orc, torch_cuda, "bf16", 14, 2, [5, 0, 63, 64, 300, 17, 90], [1, 2, 3, 40, 1, 5, 129], seed=9, min_run=min_run)


@pytest.mark.parametrize("qh,kvh", [(14, 2), (4, 4)])
@pytest.mark.parametrize("runs,length,min_run", [(255, 1, 1), (256, 1, 1), (257, 1, 1), (256, 2, 2), (352, 2, 2)])
def test_run_counts(pkv, orc, torch_cuda, qh, kvh, runs, length, min_run):
    """Around the 256 runs a block finds for itself: every run is a chunk for the prefill kernel, of one or two tokens."""
    ctx = [int(x) for x in np.random.default_rng(runs).integers(0, 150, size=runs)]
    run(pkv, orc, torch_cuda, "bf16", qh, kvh, ctx, [length] * runs, seed=runs + length, min_run=min_run)
