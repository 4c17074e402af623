"""Argument structs and what hangs on them are given back when the caller drops them."""
import gc
import weakref

import torch

from megatron_mixtera_b200 import _lib, ops


class Pool:
    """Stands for the pool tensor that a struct keeps alive."""


def test_a_launched_struct_and_its_anchor_are_freed():
    args, pool = _lib.AttentionArgs(), Pool()
    args._anchor, gone = pool, weakref.ref(pool)
    blob = ops._blob(args)
    args.num_tokens = 7  # the tensor shares the struct's memory
    assert torch.equal(blob, torch.frombuffer(bytearray(bytes(args)), dtype=torch.uint8))
    del blob, args, pool
    gc.collect()
    assert gone() is None
