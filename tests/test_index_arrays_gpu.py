"""Index arrays of a step at the batch sizes where the lengths change the way they travel: as kernel
parameters of three block sizes (up to 32, 256 and 1024 requests) and through pinned staging beyond."""
import numpy as np
import pytest
import torch

from oracle import paged_attention_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("page_size", [1, 16])
@pytest.mark.parametrize("batch", [1, 32, 33, 256, 257, 1024, 1025])
def test_index_arrays_match_the_reference_builders(batch, page_size):
    from mini_sglang_mlx_b200.attention import AttnBackend
    from mini_sglang_mlx_b200.core import Req
    from mini_sglang_mlx_b200.kernel import device_status

    class Cfg:
        head_dim, num_kv_heads = 128, 2

    rng = np.random.default_rng(batch + page_size)
    pages = rng.permutation(64 * batch).astype(np.int64)[: 6 * batch].reshape(batch, 6)
    table = (pages[:, :, None] * page_size + np.arange(page_size)).reshape(batch, -1).astype(np.int32)
    kv = rng.integers(1, table.shape[1] + 1, size=batch)
    reqs = [Req(table_idx=int(r), cached_len=int(rng.integers(0, kv[i])), device_len=int(kv[i]))
            for i, r in enumerate(rng.permutation(batch))]
    be = AttnBackend(Cfg, None, torch.from_numpy(table).cuda(), page_size=page_size)
    rows, lens = [r.table_idx for r in reqs], [r.device_len for r in reqs]
    device_status()
    pos, qo, kvp, idx, pre, mle = O.build_prefill_metadata_oracle(table, rows, [r.extend_len for r in reqs], lens)
    md = be.build_prefill_metadata(reqs)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    assert np.array_equal(host(md.positions), pos) and np.array_equal(host(md.qo_indptr), qo)
    assert np.array_equal(host(md.kv_indptr), kvp) and np.array_equal(host(md.prefix_lens), pre)
    assert np.array_equal(host(md.kv_lens), lens) and md.max_len_extend == mle
    be.split_policy = "reference"
    dm = be.build_decode_metadata(reqs)
    pos, kvp, idx, splits, mx = O.build_decode_metadata_oracle(table, rows, lens, [r.cached_len for r in reqs])
    assert np.array_equal(host(dm.positions), pos) and np.array_equal(host(dm.kv_indptr), kvp)
    assert np.array_equal(host(dm.num_kv_splits), splits) and dm.max_kv_splits == mx
    for m in (md, dm):
        if page_size == 1:
            assert np.array_equal(host(m.kv_indices), idx)
        else:
            ids = np.concatenate([pages[r, : -(-l // page_size)] for r, l in zip(rows, lens)])
            assert np.array_equal(host(m.page_indices), ids)
            assert np.array_equal(host(m.page_indptr), O.build_indptr([-(-l // page_size) for l in lens]))
    assert device_status() == 0
