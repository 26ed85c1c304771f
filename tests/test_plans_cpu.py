"""Which kept work plan a power-law product takes: host logic, with the packed store and the capture state replaced by stand-ins."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from void_b200 import _lib, _spmm, stream_k


class Tensor:
    def __init__(self, tiles):
        self.set_list(tiles)

    def set_list(self, tiles):
        self.block_rows, self.block_cols = torch.arange(tiles, dtype=torch.int32), torch.zeros(tiles, dtype=torch.int32)
        self.n_blocks = tiles


def _store(nbr=40, kind=_lib.KIND_I8):
    """A store as packing makes it: with an index of its own."""
    return SimpleNamespace(sms=148, nbr=nbr, kind=kind, row_ptr=torch.zeros(nbr + 1, dtype=torch.int32), shape=(32 * nbr, 640))


@pytest.fixture
def host(monkeypatch):
    state = SimpleNamespace(capturing=False, built=0)

    def make_plan(packed, N, np_, n_cta, mode, chunk_tiles=0, woff=None):
        state.built += 1
        plan = object.__new__(_spmm.Plan)
        plan.row_ptr, plan.tile_list, plan.shape, plan.mode = packed.row_ptr, None, packed.shape, mode
        return plan

    def workload(a):
        assert not state.capturing, "the size of a worker table is read back on the host"
        return SimpleNamespace(chunk_tiles=16, worker_offsets=None, total_work=a.n_blocks)

    monkeypatch.setattr(_spmm, "make_plan", make_plan)
    monkeypatch.setattr(stream_k, "compute_stream_k_workload", workload)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state.capturing)
    return state


TABLE = SimpleNamespace(chunk_tiles=16, worker_offsets=None)


@pytest.mark.parametrize("kind", [_lib.KIND_I8, _lib.KIND_TF32])
@pytest.mark.parametrize("tiles", [30, 100, 200])
@pytest.mark.parametrize("warm", [None, TABLE])
@pytest.mark.parametrize("captured", [None, TABLE])
def test_a_plan_of_another_tile_list_is_refused_inside_a_capture(host, kind, tiles, warm, captured):
    a = Tensor(100)
    stream_k._plan_for(a, _store(kind=kind), 256, warm, False, None)
    a.set_list(tiles)
    host.capturing = True
    with pytest.raises(_lib.VoidB200Error, match="capture"):
        stream_k._plan_for(a, _store(kind=kind), 256, captured, False, None)


@pytest.mark.parametrize("per_worker", [False, True])
def test_a_plan_of_another_tile_list_is_not_taken_outside_of_one(host, per_worker):
    a = Tensor(100)
    old = stream_k._plan_for(a, _store(), 256, TABLE, per_worker, None)
    a.block_rows[0] = 3
    store = _store()
    new = stream_k._plan_for(a, store, 256, TABLE, per_worker, None)
    assert new is not old and new.row_ptr is store.row_ptr and host.built == 2
    assert stream_k._plan_for(a, store, 256, TABLE, per_worker, None) is new


def test_worker_sums_of_another_tile_list_are_refused_inside_a_capture(host):
    a = Tensor(100)
    stream_k._plan_for(a, _store(), 256, TABLE, True, None)
    a.block_cols[3] = 1
    host.capturing = True
    with pytest.raises(_lib.VoidB200Error, match="capture"):
        stream_k._plan_for(a, _store(), 256, TABLE, True, None)


def test_a_store_of_the_same_list_takes_the_plan_that_is_kept(host):
    """Tiles edited, list and shape as they were: a store that the capture packs has another index of the same tiles."""
    a = Tensor(100)
    plan = stream_k._plan_for(a, _store(), 256, None, False, None)
    host.capturing = True
    assert stream_k._plan_for(a, _store(), 256, None, False, None) is plan
    assert stream_k._plan_for(a, _store(), 256, TABLE, False, None) is plan
    other = _store()
    other.shape = (32 * 40, 672)
    with pytest.raises(_lib.VoidB200Error, match="capture"):
        stream_k._plan_for(a, other, 256, None, False, None)
    assert host.built == 1


def test_plans_that_a_graph_reads_stay_when_a_store_of_no_graph_is_replaced():
    """One that a product packed inside a capture took, and one of a tensor that is packed for a further operand type."""
    def plan(captured):
        p = object.__new__(_spmm.Plan)
        p.captured = captured
        return p

    a, read, other = Tensor(10), plan(True), plan(False)
    a._plan_cache = {1: read, 2: other}
    _spmm.retire(a, SimpleNamespace(native=None), None)
    a._plan_cache = {}
    assert any(p is read for _, plans in a._captured_stores for p in plans)
    assert not any(p is other for _, plans in a._captured_stores for p in plans)
    _spmm.retire(a, None)
    assert len(a._captured_stores) == 1


@pytest.mark.parametrize("warm,captured", [(TABLE, None), (None, TABLE), (None, None), (TABLE, TABLE)])
@pytest.mark.parametrize("n_cta", [None, 1025])
def test_a_captured_product_finds_the_plan_of_the_other_way(host, warm, captured, n_cta):
    """From 1025 CTAs on the shares are cut along a table, which cannot be built inside a capture."""
    a, store = Tensor(100), _store()
    plan = stream_k._plan_for(a, store, 256, warm, False, n_cta)
    assert plan.mode == (1 if warm is not None or n_cta == 1025 else 3)
    host.capturing = True
    assert stream_k._plan_for(a, store, 256, captured, False, n_cta) is plan


def test_a_further_width_may_be_added_while_a_kept_plan_is_looked_for(host):
    a, store = Tensor(100), _store()
    plan = stream_k._plan_for(a, store, 256, TABLE, False, None)

    class Key(tuple):
        def __getitem__(self, i):                       # (looked at while the plans are walked)
            a._plan_cache[len(a._plan_cache)] = plan
            return tuple.__getitem__(self, i)

    a._plan_cache = {Key(("streamk", store.kind, 128, 1, 592, 1, 16)): plan, **a._plan_cache}
    host.capturing = True
    assert stream_k._plan_for(a, store, 256, None, False, None) is plan


@pytest.mark.parametrize("seed,n_cta,heavy,tiles,light", [(0, 64, 32, 100, 640), (1, 64, 4, 1000, 700), (2, 592, 40, 500, 4000), (3, 592, 300, 60, 6000),
                                                          (4, 1024, 16, 5000, 6000)])
@pytest.mark.parametrize("n_chunks", [1, 0])
def test_dealt_segments_go_where_the_least_is(seed, n_cta, heavy, tiles, light, n_chunks):
    """Few heavy rows among many light ones, several segments per CTA (which is why a piece costs four rows).  A CTA that takes a light
    row late is among the quarter with the least, so that none ends more than two light rows above the mean, unless it is by its one
    heavy segment; the same segments dealt in turn, in their order by weight, end above that."""
    from test_abi_cpu import _check_plan
    rng, cost = np.random.default_rng(seed), _spmm.ROW_COST
    cnt = rng.permutation(np.concatenate([np.full(heavy, tiles), rng.integers(1, 6, light)]))
    row_ptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    n_chunks = n_chunks or max(1, (8190 - 2 * n_cta) // len(cnt))
    segs, cptr = _check_plan(row_ptr, n_chunks, n_cta, 3, 0, cost)
    assert len(segs) >= n_cta
    costs = segs[:, 3] - segs[:, 2] + np.where(segs[:, 4] > 1, 4 * cost, cost)
    load = np.bincount(np.repeat(np.arange(n_cta), np.diff(cptr)), costs, n_cta)
    in_turn = np.bincount(np.arange(len(segs)) % n_cta, np.sort(costs)[::-1], n_cta)
    most = max(costs.max(), load.mean() + 2 * (5 + cost))
    assert load.max() <= most < in_turn.max()
