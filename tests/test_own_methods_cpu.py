"""A generate call is enqueued as one library call only while every stage method is the package's own."""

import copy
import pickle

import pytest

from dram_attention_b200 import DRAMAttention, _native
from dram_attention_b200 import dram_attention as operator_module
from dram_attention_b200 import lru_cache as cache_module
from dram_attention_b200.lru_cache import DummyCache, LRUCache
from dram_attention_b200.topk_selector import IPUpperboundTopKSelector

CHECKS = [
    (cache_module._own_cache_stages, LRUCache, ["get_kv_cache_", "_load_int32_", "update_tables_", "fetch_"]),
    (cache_module._own_selector_stages, IPUpperboundTopKSelector, ["page_list_", "score_", "select_"]),
    (operator_module._own_stages, DRAMAttention, ["attend_", "_generate_overlapped"]),
    (operator_module._own_dummy_stages, DummyCache, ["get_kv_cache_", "kv_views"]),
]


def _bare(cls):
    return cls.__new__(cls)


@pytest.mark.parametrize("own,cls,names", CHECKS, ids=[c[1].__name__ for c in CHECKS])
def test_every_replaced_stage_is_noticed(own, cls, names, monkeypatch):
    assert own(_bare(cls))
    assert own(_bare(type("Same", (cls,), {"something_else": lambda self: None})))
    assert not own(object())
    for name in names:
        assert not own(_bare(type("Traced", (cls,), {name: lambda self, *a, **k: None}))), name
        obj = _bare(cls)
        obj.__dict__[name] = lambda *a, **k: None
        assert not own(obj), name
        with monkeypatch.context() as patch:
            patch.setattr(cls, name, lambda self, *a, **k: None)
            assert not own(_bare(cls)), name
        assert own(_bare(cls))


def test_a_cache_asks_for_its_selector_too():
    cache, selector = _bare(LRUCache), _bare(IPUpperboundTopKSelector)
    cache.__dict__["top_k_selector"] = selector
    assert cache.updates_natively()
    selector.score_ = selector.score_
    assert not cache.updates_natively()
    cache.__dict__["top_k_selector"] = object()
    assert not cache.updates_natively()


def test_a_fork_is_not_copied_or_saved():
    fork = _bare(_native.Fork)
    fork.handle, fork._destroy = None, _native.lib().da_fork_destroy
    holder = {"_fork_handle": fork, "x": 1}
    assert copy.deepcopy(holder) == pickle.loads(pickle.dumps(holder)) == {"_fork_handle": None, "x": 1}
