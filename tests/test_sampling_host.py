"""What a request's sampling options are on the host: plain fields, packed beside them for the device."""
import copy
import dataclasses
import pickle
import types

import numpy as np
import pytest

from tiny_llm_b200.sampling import Sampler, SamplingParams
from tiny_llm_b200.sampling import params as packed_params, sampler as sampler_module


@pytest.mark.parametrize("again", [lambda p: SamplingParams(**vars(p)), dataclasses.replace, copy.copy, copy.deepcopy,
                                   lambda p: pickle.loads(pickle.dumps(p))])
def test_options_are_made_again_from_their_fields(again):
    """The packed row is not a field: options can be taken apart and put together, and are packed again."""
    p = SamplingParams(max_new_tokens=9, temperature=0.3, top_k=7, top_p=0.5, seed=-5, ignore_eos=True)
    q = again(p)
    assert q == p and q.packed == p.packed is not None and repr(q) == repr(p)
    assert set(vars(q)) == {f.name for f in dataclasses.fields(SamplingParams)} == set(dataclasses.asdict(q))
    with pytest.raises(dataclasses.FrozenInstanceError):
        q.seed = 1


def test_changed_options_are_packed_anew():
    p = SamplingParams(seed=3)
    assert SamplingParams(**{**vars(p), "seed": 4}).packed == SamplingParams(seed=4).packed != p.packed
    assert dataclasses.replace(p, top_k=3).packed == SamplingParams(seed=3, top_k=3).packed


def test_the_regions_of_a_block_are_the_same_packed_or_converted():
    """The options of a step reach the five regions of the host block alike from packed rows and, where one row does not
    pack (a top_k that is no int, options of another class), value by value; rows of an earlier, larger step stay behind."""
    assert packed_params.ROW.size == sampler_module._ROW.itemsize
    assert [packed_params.ROW.unpack(SamplingParams(temperature=0.1, top_p=0.2, top_k=3, seed=4).packed)] == [(0.1, 0.2, 3, 4)]
    drawn = [SamplingParams(temperature=0.3 + 0.1 * i, top_k=i, top_p=i / 8, seed=s)
             for i, s in enumerate((0, -1, -2 ** 63, 2 ** 63 - 1, 2 ** 62 + 12345, 2 ** 70 + 5))]
    rows = drawn + [SamplingParams(do_sample=False, temperature=0.0, top_k=0, top_p=1.0), SamplingParams(top_k=2 ** 31 - 1)]
    plain = [types.SimpleNamespace(**vars(p)) for p in rows]
    mixed = [SamplingParams(**{**vars(p), "top_k": float(p.top_k)}) if i == 3 else plain[i] if i == 5 else p for i, p in enumerate(rows)]
    assert mixed[3].packed is None and not hasattr(mixed[5], "packed")
    counters = [7 * i for i in range(len(rows))]
    blocks = []
    for params in (rows, plain, mixed):
        sampler = Sampler("cpu", 100, max_rows=12)
        regions = sampler._host_regions[0]
        sampler._fill(regions, 12, [SamplingParams(temperature=9.0, top_k=99, top_p=0.9, seed=99)] * 12, [999] * 12)
        sampler._fill(regions, len(params), params, counters)
        blocks.append([r.copy() for r in regions])
        whole = sampler._views(sampler._host[0], 12)          # what is copied to the device is the same memory
        assert all(np.array_equal(a, b.numpy()) for a, b in zip(regions, whole))
    n = len(rows)
    want = [np.array([p.temperature if p.do_sample else 0.0 for p in rows], "f4"), np.array([p.top_p for p in rows], "f4"),
            np.array([p.top_k for p in rows], "i4"), np.array([p.seed & (2 ** 63 - 1) for p in rows], "i8"), np.array(counters, "i8")]
    for block in blocks:
        for got, expected, old in zip(block, want, (9.0, np.float32(0.9), 99, 99, 999)):
            assert got.dtype == expected.dtype and np.array_equal(got[:n], expected) and (got[n:] == old).all()
