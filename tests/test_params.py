"""AttnParams on the host: the C struct it keeps follows the attributes, and copies are parameters of their own."""
import copy
import dataclasses
import pickle

import numpy as np

import hydra_b200 as hb
from hydra_b200 import backend


class Buffer:
    """A device buffer of another library: its address is a numpy integer."""

    def __init__(self, address):
        self.address = address

    def data_ptr(self):
        return np.int64(self.address)


def _params():
    return hb.AttnParams(q_heads=8, kv_heads=2, head_dim=64, sinks=Buffer(4096))


def test_the_struct_follows_the_attributes():
    p = _params()
    assert p.struct().sinks == 4096 and p.struct().window == 0
    p.window = 128
    p.sinks.address = 8192
    assert p.struct().window == 128 and p.struct().sinks == 8192
    p.sinks = None
    assert p.struct().sinks is None
    assert dataclasses.replace(p, window=7).struct().window == 7


def test_copies_are_parameters_of_their_own():
    p = _params()
    p.struct()                                   # the struct is there when the copy is made
    for q in (copy.copy(p), copy.deepcopy(p), pickle.loads(pickle.dumps(p))):
        assert q.struct() is not p.struct()
        q.sinks = Buffer(64)
        q.head_dim = 128
        assert (q.struct().sinks, q.struct().head_dim) == (64, 128)
        assert (p.struct().sinks, p.struct().head_dim) == (4096, 64)


def test_addresses_may_be_any_integer():
    assert backend._ptr(Buffer(4096)) == 4096 and type(backend._ptr(Buffer(4096))) is int
    assert backend._ptr(None) is None and backend._ptr(64) == 64
