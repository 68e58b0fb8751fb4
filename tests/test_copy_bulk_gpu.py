"""Block copies through the shared-memory ring: byte counts around its 8 KB pieces, fewer and more copies than
blocks in the launch, and pairs that name the same block twice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_bytes", [16, 48, 4096, 8176, 8192, 8208, 16384, 40976])
@pytest.mark.parametrize("n_pairs,n_pools", [(1, 1), (5, 2), (33, 3), (200, 13)])
def test_copies_around_the_piece_size(pkv, torch_cuda, block_bytes, n_pairs, n_pools):
    torch = torch_cuda
    rng = np.random.default_rng(block_bytes + n_pairs)
    nb = 2 * n_pairs + 3
    pools = [torch.randint(0, 256, (nb, block_bytes), dtype=torch.uint8, device="cuda") for _ in range(n_pools)]
    order = rng.permutation(nb).astype(np.int32)
    pairs = np.stack([order[:n_pairs], order[n_pairs:2 * n_pairs]], axis=1)
    pairs[::7, 1] = pairs[::7, 0]                      # nothing to do for these
    want = [p.clone() for p in pools]
    for w in want:
        w[pairs[:, 1].tolist()] = w[pairs[:, 0].tolist()]
    ptrs = torch.tensor([p.data_ptr() for p in pools], dtype=torch.int64, device="cuda")
    d_pairs = torch.from_numpy(np.ascontiguousarray(pairs)).cuda()
    pkv.launch_copy_blocks_layers(ptrs, n_pools, d_pairs, n_pairs, block_bytes)
    torch.cuda.synchronize()
    assert all(torch.equal(p, w) for p, w in zip(pools, want)) and pkv.debug_device_flags() == 0
