"""2-D views that are not contiguous, through a pipe between two contexts on one GPU: large transposed matrices, columns
of a matrix and small views, with and without a conversion, alone and beside tensors on the bulk path."""
import pytest
import torch

import tensorpipe_b200 as tpb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def link(built):
    sender, receiver = tpb.default_context("views-a"), tpb.default_context("views-b")
    listener = receiver.listen(["uv://127.0.0.1", "shm://"])
    accepted = listener.accept_future()
    out_pipe = sender.connect(listener.url("uv"))
    in_pipe = accepted.result(30)
    hello = torch.zeros(16, device="cuda")  # a pipe that is still being set up packs views first
    got, sent = in_pipe.recv(), out_pipe.send([hello], target_devices=["cuda:0"])
    got.result(30), sent.result(30)
    yield out_pipe, in_pipe
    sender.join()
    receiver.join()


def through(link, tensors, cast=None):
    out_pipe, in_pipe = link
    coming = in_pipe.recv(cast=cast or {})
    sent = out_pipe.send(tensors, target_devices=["cuda:0"] * len(tensors))
    received = coming.result(60).tensors
    sent.result(60)
    torch.cuda.synchronize()
    for i, (t, r) in enumerate(zip(tensors, received)):
        want = t.to(cast[i]) if cast and i in cast else t
        assert r.dtype == want.dtype and r.is_contiguous() and torch.equal(r, want), f"tensor {i}: {tuple(t.shape)} {t.dtype}"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int64])
@pytest.mark.parametrize("shape", [(4099, 1025), (700001, 9), (64, 70001), (2048, 2048)])
def test_large_transposed_matrices(link, dtype, shape):
    t = torch.randint(-1000, 1000, (shape[1], shape[0]), device="cuda").to(dtype).t()
    through(link, [t])
    if dtype == torch.float32:
        through(link, [t, t], cast={1: torch.bfloat16})
    through(link, [torch.randn(3 << 20, device="cuda"), t])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.uint8])
@pytest.mark.parametrize("rows,pitch,start,cols", [(16384, 1024, 256, 256), (5000, 1023, 1, 511), (30, 77, 3, 41), (300000, 24, 8, 16)])
def test_columns_of_a_matrix(link, dtype, rows, pitch, start, cols):
    t = torch.randint(0, 200, (rows, pitch), device="cuda").to(dtype)[:, start:start + cols]
    through(link, [t])
    if dtype == torch.float32:
        through(link, [t, t], cast={0: torch.bfloat16, 1: torch.float16})
    through(link, [t, torch.randn(3 << 20, device="cuda"), t.t()])


def test_an_expanded_column(link):
    t = torch.randn(1 << 20, 1, device="cuda").expand(1 << 20, 3)
    through(link, [t, t.t()])
