"""Host side of a decoder prefill: the launches it makes of a set of prompts, with the native calls recorded instead of run."""
import ctypes as C
from types import SimpleNamespace

import pytest
import torch

from rhinoforge_b200 import _native as N
from rhinoforge_b200.runtime import engine as E
from rhinoforge_b200.runtime.kv_cache import PagedKV


def ints(ptr, n):
    return torch.tensor((C.c_int32 * n).from_address(ptr)[:])


@pytest.fixture
def engine(monkeypatch):
    """An engine of chunks of 16 rows and 3 sequences per projection whose vocabulary projection answers with the row it was asked for."""
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t, *a, **k: t)
    real = N.lib()
    launches = []

    class Lib:
        def __getattr__(self, name):
            return getattr(real, name)

        def rf_stack_forward(self, handle, ref, stream):
            f = ref._obj
            launches.append(SimpleNamespace(
                tokens=f.tokens, q_start=ints(f.q_start, f.num_seqs), q_len=ints(f.q_len, f.num_seqs), kv_len=ints(f.kv_len, f.num_seqs),
                slot=ints(f.state_slot, f.num_seqs), fresh=ints(f.state_fresh, f.num_seqs), seq=ints(f.seq_of_tok, f.tokens),
                pos=ints(f.cache_pos, f.tokens), same_pos=f.pos == f.cache_pos, table=ints(f.page_table, f.num_seqs * f.pt_stride).view(f.num_seqs, -1)))
            return 0
    monkeypatch.setattr(N, "lib", lambda: Lib())
    e = object.__new__(E.DecoderEngine)
    e.device, e.dtype, e.max_tokens, e.max_batch, e.vocab_local, e.pos_stride = torch.device("cpu"), torch.float32, 16, 3, 2, 1
    e.hidden, e.cos, e.sin, e.axis, e.gdn_layers, e.handle, e.comm = torch.zeros(16, 8), torch.zeros(1), torch.zeros(1), None, [0], None, None
    e.launches, e.embedded = launches, []
    e.out_ids, e.ids, e.pos, e.kv_len = (torch.zeros(8, dtype=torch.int32) for _ in range(4))
    e.pos = e.pos[:, None]
    e.cache = PagedKV(1, 8, 72, 1, 16, device="cpu")                 # 5 pages to a sequence: no multiple of a block's four
    e._liveness, e._stream = lambda: None, lambda: None
    e._embed = lambda ids, n: e.embedded.append(ids[:n].clone())

    def head(rows, row_idx, logits_out=None):
        assert rows <= e.max_batch
        e.out_ids[:rows] = (len(launches) - 1) * 100 + row_idx[:rows]
        if logits_out is not None:
            logits_out[:] = e.out_ids[:rows, None]
    e._head = head
    yield e
    e.cache.close()


def check(e, prompts, starts, slots):
    """Every token of every prompt in one launch, in order, at its position and slot; returns the (launch, row) of each prompt's last token."""
    at, last = [0] * len(prompts), [None] * len(prompts)
    for i, (f, ids) in enumerate(zip(e.launches, e.embedded)):
        assert f.tokens <= e.max_tokens and f.same_pos and int(f.q_len.sum()) == f.tokens == ids.numel()
        for j in range(len(f.q_len)):
            s = slots.index(int(f.slot[j]))
            rows = slice(int(f.q_start[j]), int(f.q_start[j] + f.q_len[j]))
            n = int(f.q_len[j])
            assert torch.equal(ids[rows], prompts[s][at[s]:at[s] + n].int()) and bool((f.seq[rows] == j).all())
            assert f.pos[rows].tolist() == list(range(starts[s] + at[s], starts[s] + at[s] + n))
            assert int(f.fresh[j]) == (starts[s] + at[s] == 0)
            at[s] += n
            assert int(f.kv_len[j]) == starts[s] + at[s]
            own = e.cache._pt_host[slots[s]]
            assert torch.equal(f.table[j, :len(own)], own)
            # the attention kernel fetches blocks of four pages and stops at the row's end: what lies there are pages of the pool as well
            assert bool(((0 <= f.table[j]) & (f.table[j] < e.cache.num_pages)).all())
            last[s] = i * 100 + rows.stop - 1
    assert at == [p.numel() for p in prompts]
    return last


@pytest.mark.parametrize("lens,slots", [
    ([40], None),                                 # three launches of one prompt
    ([2, 1, 3, 1, 2, 4], None),                   # six prompts end in one launch, three to a projection
    ([30, 3, 5, 20, 1, 1, 1, 2], None),           # a prompt ends beside ones that begin, span and end
    ([9, 16, 7, 5, 1], [6, 2, 7, 0, 4]),          # slots out of order
])
def test_launches_of_a_prefill(engine, lens, slots):
    e = engine
    was = torch.are_deterministic_algorithms_enabled()
    torch.use_deterministic_algorithms(True)      # fresh memory holds no page number by chance
    try:
        gen = torch.Generator().manual_seed(sum(lens))
        slot_of = list(range(len(lens))) if slots is None else slots
        starts = [0] * len(lens)
        for call in range(2):                     # from empty, and behind what is there
            prompts = [torch.randint(0, 1000, (n,), generator=gen) for n in lens]
            e.launches.clear()
            e.embedded.clear()
            first, logits = e.extend(prompts, slots=slots, return_logits=True)
            last = check(e, prompts, starts, slot_of)
            assert first.tolist() == last and logits.int().tolist() == [[v, v] for v in last]
            starts = [a + n for a, n in zip(starts, lens)]
            assert [int(e.cache.lengths[s]) for s in slot_of] == starts
            if max(starts) * 2 > e.cache.max_seq_len:
                break
    finally:
        torch.use_deterministic_algorithms(was)


def test_wanted_rows_across_launches(engine):
    """Logits of chosen rows of prompts that span launches, beside the next tokens."""
    prompts = [torch.arange(n) for n in (20, 4, 15)]
    first, rows = engine.extend(prompts, slots=[3, 1, 0], want=[[0, 15, 16, 19], [], [2, 14]], return_logits=True)
    assert [r[:, 0].int().tolist() for r in rows] == [[0, 15, 100, 103], [], [110, 206]] and first.tolist() == [103, 107, 206]
