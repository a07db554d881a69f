"""What a request's sampling options are on the host: plain fields, packed beside them for the device."""
import copy
import dataclasses
import pickle

import pytest

from tiny_llm_b200.sampling import SamplingParams


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
