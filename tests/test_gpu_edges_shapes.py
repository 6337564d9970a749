"""The edge-list utilities at the edges of their forms: permutations at every bucket count and at the length where the general
sort takes over; sub_bucket with its tables in the kernel's parameters and uploaded, by counting sort and by radix sort."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 2048, 2049, 4097, 100_003, 300_001, 4_194_304, 4_194_305])
def test_randperm_is_the_order_of_the_hashes_at_every_length(n):
    """Two kernels up to 2^22 indices, the radix sort above: the same order either way -- by (44 hashed bits, index)."""
    from torchbiggraph_b200 import _C as native

    def mix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))
    seed = 123456789 + n
    h = mix(np.uint64(seed) ^ mix(np.arange(n, dtype=np.uint64) + np.uint64(0x51ED270B0F1))) >> np.uint64(20)
    want = np.lexsort((np.arange(n), h))
    for _ in range(2):                                                    # the second call uses the other counters
        np.testing.assert_array_equal(native.randperm(n, seed=seed).cpu().numpy(), want)


@pytest.mark.parametrize("rels,parts", [(1, (1, 1)), (16, (3, 5)), (17, (3, 5)), (2, (31, 33)), (2, (32, 32))])
@pytest.mark.parametrize("n", [1, 255, 1025, 20_000])
def test_sub_bucket_forms_agree_with_the_oracle(rels, parts, n):
    """Tables in the parameters (16 relations) and uploaded (17); counting sort (1023 sub-buckets) and radix sort (1024)."""
    from oracle import pbg_edges as oracle
    from torchbiggraph_b200 import _C as native
    rng = np.random.default_rng(n + rels)
    N = 700
    lhs, rhs, rel = rng.integers(0, N, n), rng.integers(0, N, n), rng.integers(0, rels, n)
    perms = [rng.permutation(N) for _ in range(2 * rels)]
    t = lambda a: torch.tensor(np.asarray(a, np.int64)).cuda()
    outs = [torch.empty(n, dtype=torch.long, device="cuda") for _ in range(3)]
    got = native.sub_bucket(t(lhs), t(rhs), t(rel), [N] * rels, [t(p) for p in perms[:rels]], [N] * rels, [t(p) for p in perms[rels:]],
                            *outs, parts[0], parts[1])
    want = oracle.sub_bucket(lhs, rhs, rel, [N] * rels, perms[:rels], [N] * rels, perms[rels:], parts[0], parts[1], False)[0]
    assert set(got) == set(want)
    for k in want:
        for x, y in zip(got[k], want[k]):
            np.testing.assert_array_equal(x.cpu().numpy(), np.asarray(y))
