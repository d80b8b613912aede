"""The allocation-free C entry point (include/tpb/noalloc.h) against the library's ordinary push kernel.

Some callers of this library cannot call cudaMalloc: a serving loop that must not trigger the
device-wide synchronisation an allocation implies, a plugin living inside a fixed memory budget, a
process whose framework already owns all device memory. For them the library exports
`tpb_noalloc_push`: its table of copies travels as the kernel's parameter (a short and a long form), and its arrive
counters are a fixed array inside the library image, which calls take in turn and leave at zero. These tests call
it through its exported C symbol (ctypes, no Python binding in between) and check that it moves
exactly the bytes the ordinary entry point moves, at the edges of both forms, and that every one of many calls
back to back publishes its flag.

This file is collected last on purpose: should it fail, a run that stops at the first failure has
already run every other test.
"""
import ctypes

import pytest
import torch

import tensorpipe_b200 as tpb
from tensorpipe_b200 import _C

MAX_ITEMS = 256


class Item(ctypes.Structure):
    _fields_ = [("src", ctypes.c_void_p), ("dst", ctypes.c_void_p), ("bytes", ctypes.c_uint64)]


def load_symbol():
    lib = ctypes.CDLL(_C.__file__)
    fn = lib.tpb_noalloc_push
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.POINTER(Item), ctypes.c_size_t, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p]
    err = lib.tpb_noalloc_strerror
    err.restype = ctypes.c_char_p
    err.argtypes = [ctypes.c_int]
    return fn, err


def ranges(rng_seed):
    """(source offset, destination offset, length) triples: empty, tiny, ragged, odd offsets, several tiles."""
    g = torch.Generator().manual_seed(rng_seed)
    sizes = [0, 1, 15, 16, 17, 4096, 8191, 8192, 8193, 70001, (1 << 20) + 3]
    out, src_off, dst_off = [], 0, 0
    for i, n in enumerate(sizes):
        skew_s = int(torch.randint(0, 16, (1,), generator=g)) if i % 2 else 0
        skew_d = int(torch.randint(0, 16, (1,), generator=g)) if i % 3 else skew_s
        out.append((src_off + skew_s, dst_off + skew_d, n))
        src_off += n + 64
        dst_off += n + 64
    return out, src_off, dst_off


@pytest.mark.gpu
def test_no_alloc_entry_point_matches_the_ordinary_kernel(built):
    fn, strerror = load_symbol()
    torch.cuda.set_device(0)
    stream = torch.cuda.current_stream().cuda_stream
    for round_index in range(2):  # the second call reuses the scratch the first one left behind
        triples, src_total, dst_total = ranges(100 + round_index)
        src = torch.randint(0, 256, (src_total,), dtype=torch.uint8, device="cuda")
        expect = torch.full((dst_total,), 0xCD, dtype=torch.uint8, device="cuda")
        got = torch.full((dst_total,), 0xCD, dtype=torch.uint8, device="cuda")
        flags = torch.zeros(4, dtype=torch.int32, device="cuda")  # [0] ordinary flag, [1] its counter, [2] new flag

        # the existing entry point
        items = [(src.data_ptr() + s, expect.data_ptr() + d, n) for s, d, n in triples]
        _C.launch_push(items, stream, True, flags.data_ptr(), 7 + round_index, flags.data_ptr() + 4)

        # the allocation-free entry point, through its C symbol
        arr = (Item * len(triples))(*[Item(src.data_ptr() + s, got.data_ptr() + d, n) for s, d, n in triples])
        rc = fn(arr, len(triples), flags.data_ptr() + 8, 7 + round_index, stream)
        assert rc == 0, strerror(rc).decode()
        torch.cuda.synchronize()

        assert torch.equal(got, expect), "the two entry points moved different bytes"
        for s, d, n in triples:
            assert torch.equal(got[d:d + n], src[s:s + n])
        assert int(flags[0]) == 7 + round_index and int(flags[2]) == 7 + round_index
        assert int(flags[1]) == 0  # the ordinary kernel leaves its counter cleared

    # requests beyond the fixed scratch are refused, with a message, and nothing is launched
    too_many = (Item * (MAX_ITEMS + 1))()
    rc = fn(too_many, MAX_ITEMS + 1, None, 0, stream)
    assert rc == -1 and b"split" in strerror(rc)
    # an empty request still publishes the flag
    rc = fn(None, 0, flags.data_ptr() + 12, 99, stream)
    assert rc == 0
    torch.cuda.synchronize()
    assert int(flags[3]) == 99


def table_of(count, g):
    """`count` non-empty ranges of ragged lengths at odd offsets, with empty ones in between where the table has room."""
    sizes = [1, 15, 16, 17, 700, 4099, 8192, 8193, 40001]
    out, src_off, dst_off = [], 0, 0
    spare = MAX_ITEMS - count
    for i in range(count):
        if spare and i % 5 == 2:
            out.append((src_off, dst_off, 0))
            spare -= 1
        n = sizes[int(torch.randint(0, len(sizes), (1,), generator=g))] + i % 3
        out.append((src_off + int(torch.randint(0, 16, (1,), generator=g)), dst_off + int(torch.randint(0, 16, (1,), generator=g)), n))
        src_off += n + 32
        dst_off += n + 48
    return out, src_off, dst_off


def push(fn, strerror, src, dst, triples, flag, value, stream):
    arr = (Item * len(triples))(*[Item(src.data_ptr() + s, dst.data_ptr() + d, n) for s, d, n in triples])
    rc = fn(arr, len(triples), flag.data_ptr(), value, stream)
    assert rc == 0, strerror(rc).decode()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 2, 15, 16, 17, 128, 255, 256])
def test_no_alloc_tables_of_every_size(built, count):
    """Both forms of the kernel, at the edges of their tables: every byte of every range and not one besides."""
    fn, strerror = load_symbol()
    stream = torch.cuda.current_stream().cuda_stream
    triples, src_total, dst_total = table_of(count, torch.Generator().manual_seed(count))
    assert len(triples) <= MAX_ITEMS and sum(n > 0 for _, _, n in triples) == count
    src = torch.randint(0, 256, (src_total,), dtype=torch.uint8, device="cuda")
    got = torch.full((dst_total,), 0xCD, dtype=torch.uint8, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    push(fn, strerror, src, got, triples, flag, count, stream)
    torch.cuda.synchronize()
    expect, from_ = torch.full((dst_total,), 0xCD, dtype=torch.uint8), src.cpu()
    for s, d, n in triples:
        expect[d:d + n] = from_[s:s + n]
    assert torch.equal(got.cpu(), expect)
    assert int(flag[0]) == count


@pytest.mark.gpu
def test_no_alloc_calls_back_to_back_publish_every_flag(built):
    """More calls than there are arrive counters (64), of several thread blocks each, in both forms: a counter that a
    call did not leave at zero would lose the flag of the call that is given it next."""
    fn, strerror = load_symbol()
    stream = torch.cuda.current_stream().cuda_stream
    calls = 200
    src = torch.randint(0, 256, (400_000,), dtype=torch.uint8, device="cuda")
    got = torch.zeros(calls, 400_000, dtype=torch.uint8, device="cuda")
    flags = torch.zeros(calls, dtype=torch.int32, device="cuda")
    for i in range(calls):
        parts = 3 if i % 3 else 20
        n = 400_000 // parts
        push(fn, strerror, src, got[i], [(k * n, k * n, n) for k in range(parts)], flags[i:], 1000 + i, stream)
    torch.cuda.synchronize()
    assert flags.tolist() == list(range(1000, 1000 + calls))
    for i in range(calls):
        whole = 400_000 // (3 if i % 3 else 20) * (3 if i % 3 else 20)
        assert torch.equal(got[i, :whole], src[:whole]) and not bool(got[i, whole:].any())
