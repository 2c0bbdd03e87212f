"""The settings of a batch of rows on their way into the kernel's buffer: the numbers that torch makes a float32 or int32 tensor of, whatever
they are given as, and its refusals."""
import warnings

import numpy as np
import pytest
import torch

from spite_b200.sampling.sampler import Sampler, SampleRow, SamplingParams


class Recorder:
    def sample(self, logits, **given):
        self.given = {k: v.clone() for k, v in given.items()}
        return torch.zeros(logits.shape[0], dtype=torch.int32)


def sample(settings, context=(5, 7), state=3):
    k = Recorder()
    rows = [SampleRow(SamplingParams(temperature=0.8, repetition_penalty=1.1), [1, 2, 3], 9),
            SampleRow(SamplingParams(**{"temperature": 0.5, "repetition_penalty": 1.2, **settings}), list(context), state)]
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        Sampler(k).sample(torch.zeros((2, 11)), rows)
    return k.given


def outcome(make):
    try:
        return make()
    except Exception:                                        # which error it is depends on who finds it
        return None


VALUES = [0, 1, 0.25, True, 40.0, 40.7, -1, 2**31 - 1, 2**31, -2**31 - 1, 2**31 - 0.5, 1e300, float("inf"), float("nan"), None, "5", np.int64(7), np.uint8(3),
          np.float32(3.0), np.float64(0.1), torch.tensor(3), torch.tensor(0.5)]


@pytest.mark.parametrize("value", VALUES, ids=repr)
@pytest.mark.parametrize("name", ["top_k", "top_p", "min_p", "temperature", "repetition_penalty", "token"])
def test_settings_as_torch_takes_them(name, value):
    kind = torch.int32 if name in ("top_k", "token") else torch.float32
    want = outcome(lambda: torch.tensor([1, value], dtype=kind)[1])
    try:
        if name == "temperature":
            value <= 0
        elif name == "repetition_penalty":
            abs(value - 1.0) < 1
    except TypeError:
        want = None                                          # the row's kind could not be told
    got = outcome(lambda: sample({}, (5, value)) if name == "token" else sample({name: value}))
    assert (got is None) == (want is None)
    if got is not None:
        got = got["context"][4] if name == "token" else got[name][1]
        assert got.dtype == kind and torch.equal(got.isnan() if want.isnan() else got, want.isnan() if want.isnan() else want)


@pytest.mark.parametrize("state", [0, 1, 2**63 - 1, 2**63, 2**64 - 1, 2**64 + 5, -1])
def test_states_as_64_bits(state):
    got = sample({}, state=state)
    assert int(got["rng_state"][1]) & (2**64 - 1) == state & (2**64 - 1) and got["context_offsets"].tolist() == [0, 3, 5]
