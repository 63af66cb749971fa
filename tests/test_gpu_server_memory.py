"""Admission counts what a session adds to the tile sets: with a budget that the
sessions' own bytes fill to the card's last percent, two sessions that fit one
by one are served one by one, and neither runs the server out of memory."""
import ctypes

import pytest

import jfcut
import synthetic

pytestmark = pytest.mark.gpu

MODEL = dict(lambda_n=100, z_weight_pct=100, lambda_t=10, k_fg=2, k_bg=2, seed_cap=1000000, kmeans_iters=32)


def trimmed_free(torch):
    """Free bytes once neither torch nor the device's pool keeps unused memory."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    rt = ctypes.CDLL("libcudart.so.12")
    pool = ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0
    return torch.cuda.mem_get_info()[0]


def test_sessions_that_fit_one_by_one(ctx):
    import torch
    torch.cuda.init()
    img, seeds = synthetic.i16_phantom(320, 320, 304, seed=3)
    srv = jfcut.Server(ctx, 0)
    try:
        sid = srv.submit(img, seeds, jfcut.PIX_I16, MODEL)
        first = srv.wait(sid)
        own = srv.stats()["used"]
    finally:
        srv.close()
    assert first.status == 0 and own > 1 << 30
    room = int(2 * own / 0.985)
    hog = torch.empty(trimmed_free(torch) - room, dtype=torch.uint8, device="cuda")
    try:
        srv = jfcut.Server(ctx, 2 * own + (1 << 20))
        try:
            sids = [srv.submit(img, seeds, jfcut.PIX_I16, MODEL) for _ in range(2)]
            for sid in sids:
                info = srv.wait(sid, 60000)
                assert info.status == 0 and info.flow == first.flow
                srv.close_session(sid)
            assert srv.stats()["peak_used"] == own
        finally:
            srv.close()
    finally:
        del hog
        torch.cuda.empty_cache()
