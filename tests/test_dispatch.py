"""Rules that send a call to one kernel or another, checked without a GPU."""
from __future__ import annotations

import re
from pathlib import Path

import torch

from kvcore_b200.kernels import api


def test_which_calls_the_tcgen05_kernel_over_rows_takes():
    """Keys and values in rows one behind the other, a positive scale, no cap, columns within 31 bits; everything else is left
    to the kernel that took it before."""
    width, page = 8 * 256, 16
    strides = (page * width, 128, width)

    def takes(dtype=torch.bfloat16, offset=0, **change):
        out = torch.empty(10 * 8 * 128 + 8, dtype=dtype)[offset:offset + 10 * 8 * 128].view(10, 8, 128)
        call = dict(value_heads=8, maps=1, key_width=128, value_width=128, page_size=page, key_strides=strides,
                    value_strides=strides, scale=0.1, softcap=None, rows_in_order=False)
        return api._rows_tc5_takes(out, **dict(call, **change))
    in_order = dict(page_size=1, key_strides=(width, 128, 0), value_strides=(width, 128, 0), rows_in_order=True)
    assert takes() and takes(torch.float32) and takes(**in_order) and takes(key_width=192)
    for scale in (0.0, -0.1, float("nan")):
        assert not takes(scale=scale)
    assert not takes(softcap=5.0) and not takes(offset=1)
    for change in (dict(key_width=64), dict(key_width=256), dict(value_width=192), dict(page_size=4), dict(page_size=128),
                   dict(value_strides=(page * width, 128, width + 8)), dict(key_strides=(page * width + 8, 128, width)),
                   dict(key_strides=(page * width, 128, 0)), dict(key_strides=(page * width, 1 << 28, width)),
                   dict(value_strides=(page * width, 1 << 28, width)), dict(maps=2, key_strides=(page * width, 1 << 27, width))):
        assert not takes(**change), change
    for change in (dict(page_size=16), dict(value_strides=(width + 8, 128, 0)), dict(key_strides=(0, 128, 0), value_strides=(0, 128, 0))):
        assert not takes(**dict(in_order, **change)), change
    assert takes(key_strides=(page * width, (1 << 28) - 8, width))


def test_the_decode_attention_waits_for_the_kernel_in_front_of_it_always():
    """What earlier kernels wrote is promised to be seen behind griddepcontrol.wait alone, and the counters that its blocks share
    may be filled right in front of it: no launch may set out as one that has waited already."""
    source = (Path(api.__file__).parent.parent / "csrc" / "attention_decode_tma.cu").read_text()
    starts = re.findall(r"bool waited = ([^;,]+)[;,]", source)
    assert starts == ["false", "false"] and len(re.findall(r"kvb_grid_wait\(\)", source)) >= 4


def test_which_experts_the_grouped_products_take(monkeypatch):
    """Matrices that no tensor map describes go the way they went before there were grouped products."""
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    x, pairs = torch.empty(500, 64, dtype=torch.bfloat16), 1000

    def matrix(*shape, offset=0):
        room = torch.empty(torch.Size(shape).numel() + 8, dtype=torch.bfloat16)
        return room[offset:offset + torch.Size(shape).numel()].view(shape)
    up, down = matrix(4, 48, 64), matrix(4, 64, 24)
    assert up.data_ptr() % 16 == 0 and down.data_ptr() % 16 == 0
    assert api.moe_path(x, pairs, 24) == api.moe_path(x, pairs, 24, up, down) == "grouped"
    for offset in (1, 2, 4):
        assert api.moe_path(x, pairs, 24, matrix(4, 48, 64, offset=offset), down) == "library"
        assert api.moe_path(x, pairs, 24, up, matrix(4, 64, 24, offset=offset)) == "library"
    many = torch.empty(1, dtype=torch.bfloat16).expand(1 << 14, 1 << 17, 64)
    assert api.moe_path(x, pairs, 1 << 16, many, down) == "library"
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert api.moe_path(x, pairs, 24, up, down) == "grouped"
    assert api.moe_path(x, pairs, 24, matrix(4, 48, 64, offset=1), down) == "tiles"
