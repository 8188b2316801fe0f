"""GPU parity tests of the device-side routing-table sort: exact order, offsets, counts and groups."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _table(rng, T, K, E, skew=False):
    if skew:
        p = 1.0 / np.arange(1, E + 1) ** 1.1
        p /= p.sum()
        return np.array([rng.choice(E, K, replace=False, p=p) for _ in range(T)], dtype=np.uint32).reshape(T, K)
    return np.array([rng.choice(E, K, replace=False) for _ in range(T)], dtype=np.uint32).reshape(T, K)


@pytest.mark.parametrize("T,K,E,skew", [(1, 8, 256, False), (8, 8, 256, False), (64, 8, 256, False), (31, 6, 64, False),
                                        (33, 3, 5, False), (4096, 8, 256, True), (2048, 6, 256, False), (1000, 1, 7, False)])
def test_device_grouping_matches_oracle(T, K, E, skew):
    import torch
    from mference_b200.moe import MoE
    rng = np.random.default_rng(T * 1000 + K)
    idx = _table(rng, T, K, E, skew)
    w = rng.integers(0, 1 << 15, (T, K)).astype(np.uint16)
    moe = MoE(d=64, f=64, num_experts=E, top_k=K, max_tokens=T, shared_bits=0)
    sp, offsets, counts, groups, n_groups = moe.encode_group(torch.from_numpy(idx.view(np.int32)).cuda(),
                                                             torch.from_numpy(w.view(np.int16)).cuda().view(torch.float16))
    pairs = np.array([(t, idx[t, r], r, w[t, r]) for t in range(T) for r in range(K)], dtype=O.PAIR_DTYPE)
    ref = O.group_pairs(pairs, T, K, E)
    got = sp.cpu().numpy().view(np.uint32)
    exp = np.stack([ref["sorted_pairs"][n] for n in ("token", "expert", "rank", "weight_bits")], axis=1)
    assert (got == exp).all()
    assert (offsets.cpu().numpy().view(np.uint32) == ref["offsets"]).all()
    assert (counts.cpu().numpy().view(np.uint32) == ref["counts"]).all()
    ng = int(n_groups.item())
    assert ng == ref["groups"].size
    g = groups.cpu().numpy().view(np.uint32)[:ng]
    assert g.tolist() == [list(map(int, x)) for x in ref["groups"].tolist()]
    # size-independent properties: a permutation of the input, sorted by (expert, token, rank)
    key = got[:, 1].astype(np.int64) * (T * K + 1) * 16 + got[:, 0].astype(np.int64) * 16 + got[:, 2]
    assert (np.diff(key) > 0).all()


def test_device_grouping_full_ragged_size_properties():
    # the ragged continuous-batch size: 86,064 rows x top-8 = 688,512 pairs; checked by properties and against the
    # host-side grouping of the library (the oracle's comparison sort is also fast enough here)
    import torch
    from mference_b200.moe import MoE
    T, K, E = 86064, 8, 256
    rng = np.random.default_rng(4)
    scores = rng.standard_normal((T, E)).astype(np.float32)
    idx = np.argsort(-scores, axis=1, kind="stable")[:, :K].astype(np.uint32)
    moe = MoE(d=64, f=64, num_experts=E, top_k=K, max_tokens=T, shared_bits=0)
    sp, offsets, counts, groups, n_groups = moe.encode_group(torch.from_numpy(idx.view(np.int32)).cuda(), None)
    got = sp.cpu().numpy().view(np.uint32)
    assert got.shape[0] == T * K
    key = got[:, 1].astype(np.int64) * (1 << 40) + got[:, 0].astype(np.int64) * 16 + got[:, 2]
    assert (np.diff(key) > 0).all()
    assert (np.bincount(got[:, 1], minlength=E) == counts.cpu().numpy().view(np.uint32)).all()
    assert (idx[got[:, 0], got[:, 2]] == got[:, 1]).all()
    assert int(counts.sum().item()) == T * K


@pytest.mark.parametrize("T,K,E", [(1, 1, 1), (33, 1, 512), (1024, 8, 256), (1025, 8, 256), (512, 16, 512), (65, 7, 37)])
def test_grouping_around_the_one_block_limit(T, K, E):
    """8192 pairs are sorted by one block, one row more by the four kernels; short last parts of a warp, most experts."""
    test_device_grouping_matches_oracle(T, K, E, False)
