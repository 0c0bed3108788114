"""What the native ``linear`` takes as its arguments (host only: CPU tensors are refused after the arguments are read)."""
import pytest
import torch

from gemmlib_b200 import ms_blkq4linear_ext as ext

NAMES = ("block_size", "col_wise", "in_features", "out_features", "input", "q_weights", "q_scales", "q_zp", "bias", "flags",
         "workspace", "out")


def values(**other):
    x = torch.zeros(2, 128, dtype=torch.float16)
    return {**dict(zip(NAMES, (64, True, 128, 32, x, *[torch.zeros(1, dtype=torch.uint8)] * 3, None, 0, False, None))), **other}


@pytest.mark.parametrize("positional", [0, 4, 11, 12])
@pytest.mark.parametrize("workspace", [None, True, False, torch.zeros(512, dtype=torch.uint8)], ids=["none", "find", "without", "tensor"])
def test_positional_and_keyword_arguments(positional, workspace):
    v = values(workspace=workspace)
    with pytest.raises(RuntimeError, match="only supports CUDA inputs"):
        ext.linear(*[v[n] for n in NAMES[:positional]], **{n: v[n] for n in NAMES[positional:]})


@pytest.mark.parametrize("change", [{"in_features": 2**32 + 128}, {"out_features": 2**40}, {"block_size": 2**64}, {"flags": 2**64},
                                    {"in_features": "128"}, {"in_features": 128.0}, {"q_zp": None}, {"input": None}, {"bias": 0}, {"out": 0}])
def test_refused_values(change):
    with pytest.raises((TypeError, OverflowError)):
        ext.linear(*values(**change).values())


def test_refused_keywords():
    v = values()
    with pytest.raises(TypeError):
        ext.linear(*list(v.values())[:11], split_k=None)
    with pytest.raises(TypeError):
        ext.linear(*list(v.values())[:11], input=v["input"])
    with pytest.raises(TypeError):
        ext.linear(*v.values(), out=None)
    with pytest.raises(TypeError):
        ext.linear(**{n: v[n] for n in NAMES[:11]})
    with pytest.raises(RuntimeError, match="Boolean value of Tensor"):
        ext.linear(*values(col_wise=torch.zeros(2)).values())
