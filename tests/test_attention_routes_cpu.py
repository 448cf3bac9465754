"""Which kernel a batch's attention goes to, and with what arguments: the launches of ``CudaOps.attention`` recorded on the CPU."""
import types

import pytest
import torch

from hcache_deepspeed_b200.inference.v2.ragged import DSStateManager, KVCacheConfig, RaggedBatchWrapper
from hcache_deepspeed_b200.inference.v2.ragged.manager_configs import DSStateManagerConfig
from hcache_deepspeed_b200.ops.backend import CudaOps


class Recorder:
    """Stands in for the kernel bindings: notes every call's name and arguments."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a, **kw: self.calls.append((name, a, kw))


def batch_of(specs, group, block=64):
    """A ragged batch of (seen, new) sequences, built for query groups of ``group``."""
    blocks = sum(-(-(s + n) // block) for s, n in specs) + 1
    cfg = DSStateManagerConfig(max_tracked_sequences=len(specs), max_ragged_batch_size=max(512, len(specs)), max_ragged_sequence_count=len(specs),
                               max_context=max(s + n for s, n in specs) + block, memory_config={"mode": "allocate", "size": blocks * block * 2 * 8 * 4})
    m = DSStateManager(cfg, (KVCacheConfig(block_size=block, cache_shape=(1, 1, 8), cache_dtype="fp32",
                                           max_blocks_per_allocation_group=-(-cfg.max_context // block)), ), device=torch.device("cpu"))
    b = RaggedBatchWrapper(cfg, block_size=block, group=group, device=torch.device("cpu"))
    for uid, (seen, new) in enumerate(specs):
        s = m.get_or_create_sequence(uid)
        s.extend_kv_cache(m.allocate_blocks(-(-(seen + new) // block)))
        s._seen_tokens = seen
        s.pre_forward(new)
        b.insert_sequence(s, torch.zeros(new, dtype=torch.int64))
    b.finalize()
    return b


def launches(batch, n_q, n_kv, d=128, dtype=torch.bfloat16, **kw):
    ops = object.__new__(CudaOps)
    ops.k = Recorder()
    q = torch.zeros(batch.current_tokens, n_q * d, dtype=dtype)
    ops.attention(q, torch.zeros_like(q), torch.zeros(1), batch, n_q, n_kv, d, 1.0, **kw)
    out = []
    for name, a, kw in ops.k.calls:
        c = types.SimpleNamespace(name=name, n_items=a[5], grouped=kw.get("grouped", False))
        if name == "paged_attention_splitkv":
            c.rows, c.splits, c.workspace = a[6], a[11], a[13]
        else:
            c.rows, c.splits, c.workspace = None, kw["n_splits"], kw["workspace"]
        out.append(c)
    return out


@pytest.mark.parametrize("n_q,n_kv", [(4, 4), (4, 2), (6, 2), (8, 2), (16, 2), (32, 2)])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
def test_rows_of_small_items(n_q, n_kv, group):
    """A batch may have been built for other groups than the attention has (a wrapper's default is 1): the kernels of few rows get
    no more than their 8, and are told of all of them; other items go to the kernel that takes 128 tokens of a head."""
    for new in range(1, 9):
        b = batch_of([(100, new), (30, 1)], group)
        calls = launches(b, n_q, n_kv)
        assert sum(c.n_items for c in calls) == 2
        for c in calls:
            if c.name == "paged_attention_splitkv":
                tokens = max(it[2] for it in b.items_small().tolist())
                assert tokens * (n_q // n_kv) <= c.rows <= 8


@pytest.mark.parametrize("n_q,n_kv", [(32, 32), (32, 8), (64, 8)])
@pytest.mark.parametrize("seqs,seen", [(40, 2000), (2, 700), (40, 100)])
def test_no_scratch_no_split(n_q, n_kv, seqs, seen):
    """Callers without scratch (the module and kernel wrappers) get unsplit launches, whatever the batch."""
    b = batch_of([(seen, 1)] * seqs, n_q // n_kv)
    assert [c.splits for c in launches(b, n_q, n_kv)] == [1]
    if seqs == 2:
        assert launches(b, n_q, n_kv, ws_small=torch.zeros(1), ws_large=torch.zeros(1))[0].splits > 1


@pytest.mark.parametrize("n_q,n_kv,d,grouped", [(32, 8, 128, True), (64, 8, 128, True), (8, 1, 128, True), (4, 4, 128, False), (8, 4, 128, False),
                                                (6, 2, 128, False), (10, 2, 128, False), (12, 2, 128, False), (14, 2, 128, False),
                                                (32, 8, 64, False), (16, 2, 64, False)])
def test_grouped_kernel_only_in_place_of_16_bit_weights(n_q, n_kv, d, grouped, monkeypatch):
    """The kernel with weights in two 16-bit parts takes the groups whose weights were 16 bits before it: 4 and 8 at 128 dims. All others,
    and all with HDS_GQA_PACKED=0, keep the kernel with fp32 weights, and its splits."""
    from hcache_deepspeed_b200.ops import backend
    ws = dict(ws_small=torch.zeros(1), ws_large=torch.zeros(1))
    for seqs, seen in ((1, 100), (3, 3000), (60, 600)):
        b = batch_of([(seen, 1)] * seqs, n_q // n_kv)
        for env in ("1", "0"):
            monkeypatch.setenv("HDS_GQA_PACKED", env)
            want = grouped and env == "1"
            c, = launches(b, n_q, n_kv, d, **ws)
            pick = backend.pick_group_splits if want else backend.pick_decode_splits
            assert c.name == "paged_attention_splitkv" and c.grouped == want and c.splits == pick(seqs, n_kv, seen + 1)
            assert c.splits == backend.pick_small_splits(seqs, n_q, n_kv, d, seen + 1)


@pytest.mark.parametrize("n_items,n_kv", [(1, 8), (4, 4), (1, 2), (9, 8)])
def test_split_counts_of_a_growing_context(n_items, n_kv):
    """Every split count is a CUDA graph of its own: a context that grows from nothing to 16384 keys passes three of them at most."""
    from hcache_deepspeed_b200.ops.backend import pick_group_splits
    counts = [pick_group_splits(n_items, n_kv, n) for n in range(1, 16385)]
    assert len(set(counts)) <= 3 and counts == sorted(counts) and max(counts) * n_items * n_kv <= 148


@pytest.mark.parametrize("rank,keys,window,want", [(512, 4096, 0, 32), (512, 8000, 0, 64), (512, 300, 0, 4), (256, 2000, 0, 16), (256, 4096, 0, 16),
                                                   (256, 4200, 0, 32), (128, 300, 0, 4), (128, 100, 0, 1), (128, 8000, 0, 32),
                                                   (128, 16000, 0, 64), (128, 16000, 4096, 32), (128, 9, 4096, 1)])
def test_splits_of_narrow_latents_get_two_tiles(rank, keys, window, want, monkeypatch):
    """Wide latents take a split per tile of 128 rows; of narrow ones more than 16 splits are as many as have two tiles."""
    from hcache_deepspeed_b200.ops import backend, kernels
    monkeypatch.setattr(kernels, "latent_attention_ctas", lambda *a: (1, 128))
    assert backend.latent_splits(1, 1, 8, rank, rank + 64, keys, window) == want
