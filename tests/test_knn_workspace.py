"""A search workspace that is sized once, for the largest batch, serves the smaller ones."""
import ctypes

import pytest
import torch

from nngpr_b200 import _lib, ops

BATCHES = [1, 7, 100, 128, 129, 500, 1000, 1183, 1184, 2000, 4000, 8000, 12000, 16000, 16383, 16384, 16385, 20000, 30000,
           40000, 65536, 100000, 300000]


def size(n_ref, n_query, d, m, f64=False):
    L = _lib.lib()
    return (L.nngp_knn_workspace_size_f64 if f64 else L.nngp_knn_workspace_size_f32)(n_ref, n_query, d, m)


@pytest.mark.parametrize('f64', [False, True])
@pytest.mark.parametrize('d,m', [(3, 32), (8, 1), (12, 32), (16, 32), (20, 32), (24, 16), (28, 32), (3, 48), (40, 32), (3, 200)])
def test_size_never_falls_with_the_queries(monkeypatch, f64, d, m):
    monkeypatch.delenv('NNGP_KNN_KERNEL', raising=False)
    for n_ref in (10, 500, 2048, 4100, 8000, 8192, 16384, 50000, 65536, 140000, 434874, 2100000):
        sizes = [size(n_ref, nq, d, m, f64) for nq in BATCHES]
        assert sizes == sorted(sizes), (n_ref, sizes)


def search(ref, q, m, ws, ws_bytes):
    out = torch.full((q.shape[0], m), -7, dtype=torch.int32, device='cuda')
    flags = ops.new_flags(ref.device)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = _lib.lib().nngp_knn_f32(p(ref), ref.shape[0], p(q), q.shape[0], ref.shape[1], None, 0, m, 0, 0, p(out), p(flags),
                                 p(ws), ws_bytes, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    _lib.check(st, 'nngp_knn_f32')
    assert int(flags.item()) == 0
    return out


@pytest.mark.gpu
@pytest.mark.parametrize('n_ref,d,largest', [(8000, 20, 40000), (16384, 12, 16384), (50000, 3, 30000), (70000, 16, 20000)])
def test_one_workspace_for_all_batches(monkeypatch, n_ref, d, largest):
    monkeypatch.delenv('NNGP_KNN_KERNEL', raising=False)
    gen = torch.Generator(device='cuda').manual_seed(n_ref)
    ref = torch.rand((n_ref, d), generator=gen, device='cuda')
    q = torch.rand((largest, d), generator=gen, device='cuda')
    bytes_ = size(n_ref, largest, d, 32)
    ws = torch.full((bytes_ + 4096,), 0xA5, dtype=torch.uint8, device='cuda')
    want = search(ref, q, 32, ws, bytes_)
    for nq in [b for b in BATCHES if b < largest]:
        assert torch.equal(search(ref, q[:nq].clone(), 32, ws, bytes_), want[:nq])
    assert bool((ws[bytes_:] == 0xA5).all())


@pytest.mark.gpu
@pytest.mark.parametrize('d,rows,per_sm', [(20, 128, 2), (16, 256, 1)])
def test_without_room_for_partial_lists_the_search_runs_unsplit(monkeypatch, d, rows, per_sm):
    monkeypatch.setenv('NNGP_KNN_KERNEL', 'tc')
    n_ref, nq = 20000, 5000
    gen = torch.Generator(device='cuda').manual_seed(d)
    ref = torch.rand((n_ref, d), generator=gen, device='cuda')
    q = torch.rand((nq, d), generator=gen, device='cuda')
    bytes_ = size(n_ref, nq, d, 32)
    room = min(-(-nq // rows) * 8, 148 * per_sm) * rows * 32 * 8
    ws = torch.full((bytes_,), 0xA5, dtype=torch.uint8, device='cuda')
    want = search(ref, q, 32, ws, bytes_)
    ws.fill_(0xA5)
    got = search(ref, q, 32, ws, bytes_ - room)
    assert torch.equal(got, want) and bool((ws[bytes_ - room:] == 0xA5).all())
    with pytest.raises(_lib.NngpError):
        search(ref, q, 32, ws, bytes_ - room - 1)
