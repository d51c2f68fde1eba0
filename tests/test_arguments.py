"""Arguments that would have a kernel read or write past a tensor are refused by the Python layer, which the native
front end hands them to (it serves only what it has found to be there).  On the CPU: nothing is launched."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.fixture()
def fp8():
    return dict(x=torch.zeros((3, 256)), w=torch.zeros((160, 256), dtype=torch.uint8), scales=torch.zeros((2, 2)), block=(128, 128),
                row0=0, k0=0, out=torch.zeros((3, 160)))


@pytest.fixture()
def moe():
    return dict(h=torch.zeros((6, 512)), route_ids=torch.zeros((3, 2), dtype=torch.int32), route_w=torch.zeros((3, 2)),
                w2=torch.zeros((4, 32, 256), dtype=torch.uint8), s2=torch.zeros((4, 32, 16), dtype=torch.uint8), e_start=0, out=None)


@pytest.mark.parametrize("change", [
    dict(scales=torch.zeros((1, 2))),                      # 160 rows need two rows of blocks
    dict(row0=112),                                        # rows 112 to 272 need three
    dict(w=torch.zeros((160, 512), dtype=torch.uint8)[:, ::2]),
    dict(out=torch.zeros((2, 160))),
    dict(out=torch.zeros((3, 160), dtype=torch.float64)),
    dict(out=torch.zeros((3, 320))[:, :160]),
])
def test_fp8_refuses(fp8, change):
    from weightstream_b200 import tp
    tp._fp8_args(**fp8)
    tp._fp8_args(**{**fp8, "row0": 96})  # the last row of the second block
    tp._fp8_args(**{**fp8, "out": torch.zeros((480,))})
    with pytest.raises(ValueError):
        tp._fp8_args(**{**fp8, **change})


@pytest.mark.parametrize("change", [
    dict(h=torch.zeros((5, 512))),
    dict(h=torch.zeros((6, 480))),
    dict(h=torch.zeros((6, 1024))[:, ::2]),
    dict(route_w=torch.zeros((3, 1))),
    dict(s2=torch.zeros((4, 32, 15), dtype=torch.uint8)),
    dict(w2=torch.zeros((4, 32, 256), dtype=torch.int16)),
    dict(out=torch.zeros((3, 31))),
])
def test_moe_refuses(moe, change):
    from weightstream_b200 import tp
    tp._moe_args(**moe)
    with pytest.raises(ValueError):
        tp._moe_args(**{**moe, **change})


@pytest.mark.gpu
def test_calls_refuse():
    """The same through the calls themselves, whose native front end looks first."""
    from weightstream_b200 import tp
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    dev = torch.device("cuda:0")
    ep = tp.Endpoint(max_m=8, max_n=160, max_vocab=160)
    w, sc, x = torch.zeros((160, 256), dtype=torch.uint8, device=dev), torch.ones((2, 2), device=dev), torch.zeros((3, 256), device=dev)
    short = sc[:1]
    bits = np.zeros((3, 256), np.uint16)
    w2, s2 = torch.zeros((4, 32, 256), dtype=torch.uint8, device=dev), torch.zeros((4, 32, 16), dtype=torch.uint8, device=dev)
    ids, rw = torch.zeros((3, 2), dtype=torch.int32, device=dev), torch.zeros((3, 2), device=dev)
    try:
        for call in (lambda: ep.fp8_rowpar_gemm_allreduce(x, w, short),
                     lambda: ep.fp8_rowpar_gemm_allreduce(x, w, sc, out=torch.zeros((2, 160), device=dev)),
                     lambda: ep.lm_head_allgather_argmax(x, w, short, vocab_row0=0, vocab=160),
                     lambda: ep.fp8_rowpar_gemm_allreduce_host(bits[:, :255], w, sc),
                     lambda: ep.fp8_rowpar_gemm_allreduce_host(bits, w, sc, x_dtype=tp.WS_ACT_F32),
                     lambda: ep.fp8_rowpar_gemm_allreduce_host(bits, w, short),
                     lambda: ep.moe_down_combine_allreduce(torch.zeros((5, 512), device=dev), ids, rw, w2, s2, 0),
                     lambda: ep.moe_down_combine_allreduce(torch.zeros((6, 512), device=dev), ids, rw, w2, s2[:3].contiguous(), 0)):
            with pytest.raises(ValueError):
                call()
        assert ep.launches == 0
        ep.fp8_rowpar_gemm_allreduce(x, w, sc)
        ep.fp8_rowpar_gemm_allreduce_host(bits.view(np.uint8), w, sc)  # bytes that hold what is needed
        ep.moe_down_combine_allreduce(torch.zeros((6, 512), device=dev), ids, rw, w2, s2, 0)
        ep.check()
    finally:
        ep.close()
