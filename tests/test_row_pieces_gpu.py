"""Results in rows without 16-byte alignment, written as aligned 32-byte pieces that span the sixteen columns an epilogue step has and those before them: every distance of
a row from a piece's boundary (odd N and ldc, destinations that begin in the middle of one), every length of the last columns, tiles of every form, in bf16, f32 and s32,
against exact products; what lies between the rows and behind them stays as it was."""
import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

TORCH = {"bf16": "bfloat16", "f32": "float32", "s32": "int32"}


@pytest.mark.parametrize("dt", ["bf16", "f32", "s32"])
@pytest.mark.parametrize("M,N", [(200, n) for n in (1, 3, 15, 17, 31, 33, 63, 65, 95, 127, 129, 130, 255, 257, 500, 501)] + [(600, 3001), (2300, 1029)])
@pytest.mark.parametrize("pad,start", [(0, 0), (3, 1), (8, 5), (1, 7)])
def test_every_distance_from_a_boundary(capi, monkeypatch, dt, M, N, pad, start):
    import torch
    torch.manual_seed(N + pad)
    K, ldc = 160, N + pad
    a, w = (torch.randint(-9, 10, s, dtype=torch.int8, device="cuda") for s in ((M, K), (K, N)))
    want = (a.float() @ w.float()).to(getattr(torch, TORCH[dt]))
    pool = torch.full((start + M * ldc + 40,), 77, dtype=want.dtype, device="cuda")
    out = pool[start:start + M * ldc].view(M, ldc)
    for pair, split in (("0", "1"), ("0", "2"), ("1", "0")):       # one CTA a tile, a tile's K shared by two, pairs of CTAs
        monkeypatch.setenv("B200DNN_TC_PAIR", pair)
        monkeypatch.setenv("B200DNN_TC_KSPLIT", split)
        pool.fill_(77)
        d = capi.make_matmul(M, N, K, a, w, out, src_dt=capi.DT["s8"], dst_dt=capi.DT[dt], force_kernel=2, ldc=ldc)
        capi.check(capi.matmul(d, torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(out[:, :N], want), (dt, N, pad, start, pair, split)
        assert (pool[:start] == 77).all() and (pool[start + M * ldc:] == 77).all() and (out[:, N:] == 77).all()
    capi.lib.b200dnn_clear_caches()
