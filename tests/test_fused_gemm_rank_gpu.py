"""The GEMMs that are fused with a collective, as rank 1 of 2 launches them: tiles rotate so that what is local comes first.
Two allocations of one GPU stand for the arenas of both ranks, and all that the other rank would send lies there before the
launch, so that nothing is waited for but the launch's own copies. In a child process, because the arena is one per process."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent("""
    import ctypes as C, sys, torch
    sys.path.insert(0, %r)
    import tensorplay_b200.ops as O
    from tensorplay_b200 import _native
    from tensorplay_b200.ops._common import status_word, stream_ptr
    from tensorplay_b200.parallel import tp

    form, M, N, K = sys.argv[1], *map(int, sys.argv[2:])
    W, RANK, PAD, EPOCH = 2, 1, 4096, 1
    READY, DONE, CNT = 0, 2, 4
    torch.manual_seed(M + N + K)
    x, w = (torch.randn(n, K, device="cuda").bfloat16() for n in (M, N))
    bias = torch.randn(N, device="cuda").bfloat16()
    gathered = {"rows": x, "weight": w, "reduce": torch.empty(M * N, dtype=torch.bfloat16)}[form]
    size = PAD + 2 * gathered.numel()
    arenas = [torch.full((size // 2,), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(W)]
    pads = [a.view(torch.int32)[:PAD // 4] for a in arenas]
    body = [a[PAD // 2:].view(gathered.shape) for a in arenas]
    for p in pads:
        p.zero_()
    _native.kernels()
    raw = C.CDLL(str(_native._LIBDIR / "libtpb200.so"))
    _native.register_sigs(raw, tp._SIGS)
    adopt = raw._ZN3tpb10symm_adoptEiiPKPcmS0_   # tpb::symm_adopt: mapped arenas become the process's symmetric memory
    adopt.argtypes, adopt.restype = [C.c_int, C.c_int, C.POINTER(C.c_void_p), C.c_size_t, C.c_void_p], None
    adopt(W, RANK, (C.c_void_p * W)(*(a.data_ptr() for a in arenas)), size, None)
    st, s = status_word(x.device).data_ptr(), stream_ptr()
    flags = torch.zeros(1024, dtype=torch.int32, device="cuda")
    ref = x.double() @ w.double().t()
    mag = x.double().abs() @ w.double().abs().t() * K * 2.0 ** -24   # of adding K products in fp32

    if form == "reduce":
        out = torch.full((M // W, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        stage = [b.view(W, M // W, N) for b in body]
        other = torch.randn(M // W, N, device="cuda").bfloat16()
        stage[RANK][0] = other
        tiles = (M + 127) // 128 * ((N + 255) // 256)
        cols = 128 if N <= 128 or 2 * tiles <= torch.cuda.get_device_properties(0).multi_processor_count else 256
        pads[RANK][CNT] = M // W // 32 * ((N + cols - 1) // cols)   # all tiles of rank 0 have arrived
        code = raw.tpb_gemm_rs(x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, K, K, 0, 0, PAD, 0, CNT, EPOCH, 5.0, st, s, None)
        assert code == 0, code
        O.check_status()
        torch.cuda.synchronize()
        # partial rows are rounded to bf16, and so is their sum
        sent, own = stage[0][RANK].double(), ref[M // W:] + other.double()
        assert ((sent - ref[:M // W]).abs() <= ref[:M // W].abs() * 2.0 ** -8 + mag[:M // W]).all()
        assert ((out.double() - own).abs() <= (ref[M // W:].abs() + own.abs()) * 2.0 ** -8 + mag[M // W:]).all()
        assert pads[0][CNT + RANK].item() == pads[RANK][CNT + RANK].item() == pads[RANK][CNT].item()
    else:
        out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        n = gathered.shape[0] // W
        for r in range(W):
            body[r][r * n:(r + 1) * n] = gathered[r * n:(r + 1) * n]
        pads[RANK][READY] = EPOCH   # rank 0's shard is there
        if form == "rows":
            code = raw.tpb_ag_gemm(PAD, w.data_ptr(), out.data_ptr(), bias.data_ptr(), M, N, K, K, N, 0, 0, flags.data_ptr(), 64, 0,
                                   READY, DONE, EPOCH, 4, 5.0, st, s, None)
        else:
            code = raw.tpb_ag_gemm_weight(x.data_ptr(), PAD, out.data_ptr(), bias.data_ptr(), M, N, K, K, N, 0, 0, flags.data_ptr(),
                                          64, 0, READY, DONE, EPOCH, 4, 5.0, st, s, None)
        assert code == 0, code
        O.check_status()
        torch.cuda.synchronize()
        ref += bias.double()
        assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + mag).all()
        assert torch.equal(body[RANK], gathered)
        for p in pads:   # told to both: the shards may be written again, and rank 1's shard was there
            assert p[DONE + RANK].item() == EPOCH and p[READY + RANK].item() == EPOCH
    print("OK")
""") % ROOT


# tiles of 256 columns, of 128, and a shard that is no whole number of tiles (no rotation)
@pytest.mark.parametrize("form", ["rows", "weight", "reduce"])
@pytest.mark.parametrize("M,N,K", [(1024, 2560, 320), (512, 1024, 256), (384, 640, 200)])
def test_as_rank_1_of_2(form, M, N, K):
    out = subprocess.run([sys.executable, "-c", CHILD, form, str(M), str(N), str(K)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout + out.stderr
