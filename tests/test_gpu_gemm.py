"""Parity of the two GEMM kernels against the CPU oracle (through the Python shim, i.e. the C ABI)."""
import numpy as np
import pytest
import torch

import oracle
from helpers import check_gemm_sampled, check_gemm_tolerance, make_packed, make_x, to_dev

pytestmark = pytest.mark.gpu

_cache = {}


def packed(N, K, g):
    key = (N, K, g)
    if key not in _cache:
        _cache[key] = make_packed(N, K, g, seed=1234 + N % 97 + K % 89)
    return _cache[key]


def run(M, N, K, g, algo, bias=False, seed=4321):
    import quant
    p = packed(N, K, g)
    qw, zs = to_dev(p)
    x = make_x(M, K, seed)
    b = None
    if bias:
        gen = torch.Generator().manual_seed(5)
        b = (torch.randn(1, N, generator=gen) * 0.02).half()
    out = quant.gemm_awq_bias(x.cuda(), qw, zs, None if b is None else b.cuda(), N, g, algo=algo)
    torch.cuda.synchronize()
    ref = oracle.gemm_f16(x, p["w_deq"], None if b is None else b)
    assert out.shape == (1, M, N)
    return check_gemm_tolerance(out[0], ref.astype(np.float32), x, p["w_deq"], K)


SKINNY_SHAPES = [(64, 128, 128), (96, 256, 64), (32, 32, 32), (4096, 1024, 128), (1376, 1408, 64), (512, 4096, 128),
                 (4096, 512, 128), (160, 1344, 64)]


@pytest.mark.parametrize("N,K,g", SKINNY_SHAPES)
@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 16, 17, 32])
def test_skinny_small_tokens(N, K, g, M):
    run(M, N, K, g, algo=1, bias=(M % 2 == 0))


@pytest.mark.parametrize("N,K,g", [(1536, 4096, 64), (2752, 4096, 64), (512, 11008, 64), (1024, 16384, 128)])
@pytest.mark.parametrize("M", [24, 32])
def test_decode_kernel_17_to_32_tokens_cluster_shapes(M, N, K, g):
    """17..32 tokens: the launch shape is searched over cluster sizes 1..8 (odd ones included) or falls back to
    two 16-token passes; these shapes hit 3-, 7/8-CTA clusters and the fallback."""
    run(M, N, K, g, algo=1, bias=True)


@pytest.mark.parametrize("M", [33, 100, 257])
def test_skinny_many_tokens_fallback(M):
    run(M, 256, 512, 128, algo=1, bias=True)


@pytest.mark.parametrize("K,N", [(4096, 4096), (4096, 16384), (16384, 4096)])
@pytest.mark.parametrize("M", [1, 4, 8, 16])
def test_skinny_opt_shapes(K, N, M):
    """The decode sweep of the benchmark: every (shape, M) against the full oracle product."""
    run(M, N, K, 128, algo=1)


@pytest.mark.parametrize("wn,splits", [(1, 1), (1, 8), (2, 4), (4, 2), (8, 1), (8, 8), (2, 1), (16, 1), (16, 4)])
def test_skinny_every_decomposition(wn, splits):
    """The 16-warp decode kernel (17..32 tokens by default), forced onto small token counts too."""
    import quant
    lib = quant.load_library()
    try:
        lib.w4a16_tune_decode(1, 0, 0, 0)
        lib.w4a16_tune_skinny(wn, splits)
        run(5, 256, 2048, 128, algo=1, bias=True)
        run(16, 96, 1344, 64, algo=1)
        run(24, 256, 2048, 128, algo=1, bias=True)
    finally:
        lib.w4a16_tune_skinny(0, 0)
        lib.w4a16_tune_decode(0, 0, 0, 0)


@pytest.mark.parametrize("tn", [1, 2, 4, 8])
@pytest.mark.parametrize("splits", [1, 2, 3, 4, 8])
def test_gemv_every_decomposition(tn, splits):
    """The 8-warp decode kernel over its launch shapes: out-feature tiles per CTA x cluster size x ring depth, with
    every activation box height (1, 2, 4, 8, 16 rows), a K that is not a multiple of the 128-k unit, group sizes
    32/64/128 and an out-feature count that leaves the last CTA partly empty."""
    import quant
    lib = quant.load_library()
    ran = 0
    try:
        for depth in (2, 3, 0):
            lib.w4a16_tune_decode(2, tn, splits, depth)
            for (M, N, K, g) in [(1, 256, 2048, 128), (2, 160, 1344, 64), (3, 256, 2048, 128), (5, 256, 2048, 128),
                                 (8, 96, 1024, 32), (12, 160, 1344, 64), (16, 256, 2048, 128)]:
                try:
                    run(M, N, K, g, algo=1, bias=(M % 2 == 1))
                    ran += 1
                except RuntimeError as e:
                    if "algo" not in str(e):
                        raise                                    # only "this shape cannot run with the forced decomposition"
    finally:
        lib.w4a16_tune_decode(0, 0, 0, 0)
    if ran == 0:
        pytest.skip("no test shape can run with this forced decomposition (fewer 128-k units than K slices)")
    flag = __import__("ctypes").c_int(-1)
    assert lib.w4a16_device_error_flag(flag) == 0 and flag.value == 0


def test_gemv_more_than_sixteen_tokens_in_passes():
    """Forced onto the 8-warp kernel, 17+ tokens run as passes of 16 over gridDim.z."""
    import quant
    lib = quant.load_library()
    try:
        lib.w4a16_tune_decode(2, 0, 0, 0)
        run(17, 256, 2048, 128, algo=1, bias=True)
        run(40, 160, 1344, 64, algo=1)
    finally:
        lib.w4a16_tune_decode(0, 0, 0, 0)


def test_identity_trick_reads_back_the_dequantised_weight():
    """x = I  =>  out[k, n] = w[n, k] exactly (one product, fp32 -> fp16 is exact for an fp16 value)."""
    import quant
    N, K, g = 96, 256, 64
    p = packed(N, K, g)
    qw, zs = to_dev(p)
    eye = torch.eye(K, dtype=torch.float16, device="cuda").unsqueeze(0)
    for algo in (1, 2):
        out = quant.gemm_awq_bias(eye, qw, zs, None, N, g, algo=algo)
        got = out[0].t().contiguous().cpu().numpy().view(np.uint16).copy()
        exp = p["w_deq"].view(np.uint16).copy()
        got[(got & 0x7FFF) == 0] = 0
        exp[(exp & 0x7FFF) == 0] = 0
        assert np.array_equal(got, exp), f"algo {algo}"


TC_SHAPES = [(128, 128, 128), (128, 256, 64), (256, 512, 128), (96, 256, 64), (1376, 1408, 64), (4096, 1024, 128)]


@pytest.mark.parametrize("N,K,g", TC_SHAPES)
@pytest.mark.parametrize("M", [33, 64, 100, 128, 200, 256, 300, 511, 513])
def test_tc_parity(N, K, g, M):
    run(M, N, K, g, algo=2, bias=(M % 2 == 1))
    import quant
    flag = __import__("ctypes").c_int(-1)
    assert quant.load_library().w4a16_device_error_flag(flag) == 0 and flag.value == 0


@pytest.mark.parametrize("tile", [64, 128, 256])
def test_tc_every_token_tile(tile):
    import quant
    lib = quant.load_library()
    try:
        lib.w4a16_tune_tc(tile, 0)
        run(300, 384, 1024, 128, algo=2, bias=True)
        run(1, 128, 128, 128, algo=2)
    finally:
        lib.w4a16_tune_tc(0, 0)


@pytest.mark.parametrize("tile,split", [(256, 2), (128, 2), (128, 4), (64, 4)])
def test_tc_split_k(tile, split):
    """K split over several CTAs per output tile: fp32 partials through the workspace, summed in a fixed
    order by the last arriver - parity, determinism, counters left at zero for the next call."""
    import quant
    lib = quant.load_library()
    try:
        lib.w4a16_tune_tc(tile, split)
        for _ in range(2):                                   # second call reuses self-reset counters
            run(300, 384, 2048, 128, algo=2, bias=True)
        run(70, 1376, 1408, 64, algo=2)
        p = packed(384, 2048, 128)
        qw, zs = to_dev(p)
        x = make_x(300, 2048).cuda()
        a = quant.gemm_awq_bias(x, qw, zs, None, 384, 128, algo=2)
        b = quant.gemm_awq_bias(x, qw, zs, None, 384, 128, algo=2)
        assert torch.equal(a, b)
    finally:
        lib.w4a16_tune_tc(0, 0)
    flag = __import__("ctypes").c_int(-1)
    assert lib.w4a16_device_error_flag(flag) == 0 and flag.value == 0


def test_tc_bert_ffn_up_config():
    """M=512 (4 x 128), K=1024, N=4096, g=128."""
    run(512, 4096, 1024, 128, algo=0, bias=True)


@pytest.mark.parametrize("K,N", [(4096, 4096), (4096, 16384), (16384, 4096)])
def test_tc_opt_shapes_linearity(K, N):
    """Full-size property check (the oracle would take minutes): f(x1 + x2) ~= f(x1) + f(x2) and
    agreement with an fp16 cuBLAS matmul on the bit-exact dequantised weight."""
    import quant
    g, M = 128, 2048
    gen = torch.Generator().manual_seed(N + K)
    w = (torch.randn(N, K, generator=gen) * 0.02).half().cuda()
    from w4a16 import quant_lmdeploy
    qw, zs, _ = quant_lmdeploy(w, K, N, g, 4)
    wd = quant.dequant(qw, zs, N, K, g)
    x = torch.randn(1, M, K, generator=gen).half().cuda()
    out = quant.gemm_awq_bias(x, qw, zs, None, N, g, algo=2)
    ref = (x[0].float() @ wd.float().t())
    fro = ((out[0].float() - ref).norm() / ref.norm()).item()
    assert fro <= 2e-3, fro
    err = (out[0].float() - ref).abs().max().item()
    assert err <= 1e-2 * x.abs().max().item() * (K ** 0.5) * wd.abs().max().item()


@pytest.mark.parametrize("K,N", [(4096, 4096), (4096, 16384), (16384, 4096)])
@pytest.mark.parametrize("M", [512, 8192])
def test_tc_opt_shapes_sampled_oracle(K, N, M):
    """The prefill sweep of the benchmark through the plan the library selects (workspace from
    w4a16_workspace_bytes, i.e. the split-K plan where it chooses one), against the oracle on a seeded sample of
    16 token rows x 48 out-features."""
    import quant
    p = packed(N, K, 128)
    qw, zs = to_dev(p)
    x = make_x(M, K, seed=7 + M)
    out = quant.gemm_awq_bias(x.cuda(), qw, zs, None, N, 128, algo=0)
    torch.cuda.synchronize()
    check_gemm_sampled(out[0], x, p)
    flag = __import__("ctypes").c_int(-1)
    assert quant.load_library().w4a16_device_error_flag(flag) == 0 and flag.value == 0


@pytest.mark.parametrize("K,N", [(4096, 11008), (11008, 4096), (4096, 4096)])
@pytest.mark.parametrize("M", [16, 32, 1024])
def test_llama_shapes_group64_sampled_oracle(K, N, M):
    """LLaMA-2-7B-shaped linears at group size 64, unsharded: decode at 16 and 32 tokens, prefill at 1024."""
    import quant
    p = packed(N, K, 64)
    qw, zs = to_dev(p)
    x = make_x(M, K, seed=11 + M)
    out = quant.gemm_awq_bias(x.cuda(), qw, zs, None, N, 64, algo=0)
    torch.cuda.synchronize()
    check_gemm_sampled(out[0], x, p, n_tok=16, n_out=48)


def test_api_contract_errors():
    import quant
    p = packed(64, 128, 128)
    qw, zs = to_dev(p)
    x = make_x(4, 128).cuda()
    with pytest.raises(RuntimeError, match="dimension"):
        quant.gemm_awq_ut(x[0], qw, zs, 4, 64, 128, 128)
    with pytest.raises(RuntimeError, match="contiguous"):
        quant.gemm_awq_ut(x.transpose(1, 2).contiguous().transpose(1, 2), qw, zs, 4, 64, 128, 128)
    with pytest.raises(RuntimeError, match="dtype"):
        quant.gemm_awq_ut(x.float(), qw, zs, 4, 64, 128, 128)
    with pytest.raises(RuntimeError, match="CUDA"):
        quant.gemm_awq_ut(x.cpu(), qw, zs, 4, 64, 128, 128)
    with pytest.raises(RuntimeError):
        quant.gemm_awq_ut(x, qw, zs, 4, 64, 128, 100)          # unsupported group size
    with pytest.raises(RuntimeError):
        quant.gemm_awq_ut(x, qw, zs, 4, 48, 128, 128)          # N not a multiple of 32 / wrong sizes
    # M and K arguments are ignored like in the reference (gemm_quant.cu:85-87)
    a = quant.gemm_awq_ut(x, qw, zs, 12345, 64, 999, 128)
    b = quant.gemm_awq_ut(x, qw, zs, 4, 64, 128, 128)
    assert torch.equal(a, b)


def test_output_canaries_and_determinism():
    """Nothing is written outside [tokens, N]; repeated calls give identical bits."""
    import quant
    lib = quant.load_library()
    N, K, g = 160, 1344, 64
    p = packed(N, K, g)
    qw, zs = to_dev(p)
    for M, algo in [(5, 1), (16, 1), (70, 2), (300, 2)]:
        x = make_x(M, K).cuda()
        big = torch.full((M + 2, N), 777.0, dtype=torch.float16, device="cuda")
        out = big[1:M + 1]
        st = lib.w4a16_gemm_algo(x.data_ptr(), qw.data_ptr(), zs.data_ptr(), None, out.data_ptr(), M, N, K, g,
                                 None, 0, torch.cuda.current_stream().cuda_stream, algo)
        assert st == 0
        torch.cuda.synchronize()
        assert (big[0] == 777.0).all() and (big[M + 1] == 777.0).all()
        again = quant.gemm_awq_bias(x, qw, zs, None, N, g, algo=algo)
        assert torch.equal(again[0], out)


def test_non_default_stream_and_graph_replay():
    import quant
    N, K, g = 512, 4096, 128
    p = packed(N, K, g)
    qw, zs = to_dev(p)
    for M, algo in [(8, 1), (256, 2)]:
        x = make_x(M, K).cuda()
        eager = quant.gemm_awq_bias(x, qw, zs, None, N, g, algo=algo)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            side = quant.gemm_awq_bias(x, qw, zs, None, N, g, algo=algo)
        s.synchronize()
        assert torch.equal(eager, side)
        out = torch.empty_like(eager)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            quant.gemm_awq_bias(x, qw, zs, None, N, g, algo=algo, out=out)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(eager, out)


def test_static_weights_flag_dependent_chain():
    """W4A16_FLAG_STATIC_WEIGHTS (programmatic dependent launch): a chain in which every call consumes
    the previous call's output gives the same bits as the plain launches, eagerly and in a CUDA graph."""
    import quant
    N = K = 1024
    g = 128
    ps = [make_packed(N, K, g, seed=50 + i) for i in range(3)]
    devs = [to_dev(p) for p in ps]
    x = (make_x(4, K) * 0.5).cuda()

    def chain(static, bufs=None):
        h = x
        for i in range(6):
            qw, zs = devs[i % 3]
            h = quant.gemm_awq_bias(h, qw, zs, None, N, g, static_weights=static, out=None if bufs is None else bufs[i])
        return h

    plain = chain(False)
    pdl = chain(True)
    assert torch.equal(plain, pdl)
    bufs = [torch.empty(1, 4, N, dtype=torch.float16, device="cuda") for _ in range(6)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(True, bufs)
    for b in bufs:
        b.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(bufs[5], plain)


def test_walinear_module_and_host_buffer_entry_point():
    import ctypes
    import quant
    from w4a16 import WALinear
    lin = torch.nn.Linear(256, 128, bias=True).half().cuda()
    q = WALinear.from_float(lin, {"n_bit": 4, "group_size": 128})
    assert q.weight.dtype == torch.int32 and tuple(q.weight.shape) == (256, 16)
    assert tuple(q.zeros_scales.shape) == (2, 256) and tuple(q.bias.shape) == (1, 128)
    x = torch.randn(2, 3, 256, dtype=torch.float16, device="cuda")
    y = q(x)
    wd = quant.dequant(q.weight, q.zeros_scales, 128, 256, 128)
    ref = (x.float() @ wd.float().t()).half() + lin.bias.data.half()
    assert torch.allclose(y.float(), ref.float(), atol=2e-2, rtol=2e-2)
    # state-dict round trip with the reference's buffer names
    sd = q.state_dict()
    assert set(sd) == {"zeros_scales", "weight", "bias"}
    q2 = WALinear(256, 128, w_bit=4, group_size=128, bias=True)
    q2.load_state_dict(sd)
    assert torch.equal(q2(x), y)
    # host-buffer C-ABI call
    lib = quant.load_library()
    M = 6
    xh = x.reshape(M, 256).cpu().pin_memory()
    oh = torch.empty(M, 128, dtype=torch.float16).pin_memory()
    xd = torch.empty(M, 256, dtype=torch.float16, device="cuda")
    od = torch.empty(M, 128, dtype=torch.float16, device="cuda")
    st = lib.w4a16_gemm_host(xh.data_ptr(), oh.data_ptr(), xd.data_ptr(), od.data_ptr(), q.weight.data_ptr(),
                             q.zeros_scales.data_ptr(), q.bias.data_ptr(), M, 128, 256, 128, None, 0,
                             torch.cuda.current_stream().cuda_stream)
    assert st == 0
    assert torch.equal(oh, y.reshape(M, 128).cpu())


@pytest.mark.parametrize("blocks,splits", [(0, 0), (1, 1), (1, 3), (2, 2), (3, 1), (2, 8)])
def test_narrow_every_decomposition(blocks, splits):
    """The batched-decode kernel over its launch shapes: out-feature blocks per cluster x cluster size, every token tile
    (16 / 32 / 64) at its edges, both group sizes, a K that is not a multiple of the 128-k stage, and out-feature counts
    that leave a block partly and a cluster's last block wholly empty."""
    import quant
    lib = quant.load_library()
    try:
        lib.w4a16_tune_decode(3, blocks, splits, 0)
        for (M, N, K, g) in [(1, 96, 1344, 64), (9, 416, 2048, 128), (16, 416, 1344, 64), (17, 96, 1024, 128), (24, 416, 2048, 128),
                             (32, 1376, 1408, 64), (33, 416, 1344, 64), (64, 416, 2048, 128)]:
            run(M, N, K, g, algo=0, bias=(M % 2 == 1))
    finally:
        lib.w4a16_tune_decode(0, 0, 0, 0)
    flag = __import__("ctypes").c_int(-1)
    assert lib.w4a16_device_error_flag(flag) == 0 and flag.value == 0


def test_narrow_is_no_less_exact_than_the_decode_kernels_and_keeps_their_epilogues():
    """The scale is applied in fp32 to exact integer sums: with fp16 rounding of the output only (2^-11 relative to each
    output, plus fp32 sums) against float64; residual and SwiGLU epilogues round like the launches they replace."""
    import quant
    lib = quant.load_library()
    for (M, n, K, g) in [(9, 704, 1024, 64), (24, 512, 4096, 128), (32, 2752, 4096, 64)]:
        N = 2 * n
        p = packed(N, K, g)
        qw, zs = to_dev(p)
        x = make_x(M, K)
        q = lambda **kw: quant.gemm_awq_bias(x.cuda(), qw, zs, None, N, g, **kw)
        r = torch.randn(1, M, N, generator=torch.Generator().manual_seed(3)).half().cuda()
        outs = {}
        try:
            for kernel in (1, 3):
                lib.w4a16_tune_decode(kernel, 0, 0, 0)
                plain, res = q(), q(residual=r)
                silu = q(silu_mul=True)
                assert torch.equal(res, plain + r)
                assert torch.equal(silu, quant.silu_mul_tiles(plain))
                outs[kernel] = plain[0].double().cpu()
        finally:
            lib.w4a16_tune_decode(0, 0, 0, 0)
        z = torch.from_numpy(p["zs"].view(np.float16).astype(np.float64)).reshape(K // g, N, 2)
        codes = quant.dequant(qw, torch.stack((torch.full((K // g, N), 64.0), torch.ones(K // g, N)), -1).half().reshape(K // g, 2 * N).cuda(), N, K, g)
        w = (codes.double().cpu().reshape(N, K // g, g) - (z[..., 0].t()[..., None] - 64.0)) * z[..., 1].t()[..., None]
        ref = x[0].double() @ w.reshape(N, K).t()
        err = {k: ((o - ref).norm() / ref.norm()).item() for k, o in outs.items()}
        assert err[3] <= 1.02 * err[1] and err[3] <= 2.0 ** -11, err       # an fp16 rounding is at most 2^-11 of each output


@pytest.mark.parametrize("M,N,K,g,kernel", [
    (8, 512, 1024, 64, "decode"), (9, 512, 1024, 64, "batched"), (16, 512, 1024, 128, "decode"), (17, 512, 1024, 128, "batched"),
    (32, 512, 1024, 64, "batched"), (33, 512, 1024, 64, "batched"), (64, 512, 2048, 128, "batched"), (65, 512, 1024, 64, "prefill"),
    # 33 to 64 tokens go to the kernel that is faster there: wide matrices and a short K with groups of 64 to the prefill kernel
    (48, 4096, 2048, 128, "batched"), (33, 9472, 4096, 128, "batched"), (48, 11008, 1024, 64, "prefill"), (48, 11008, 4096, 64, "prefill"),
    (64, 9600, 768, 128, "prefill"), (40, 12256, 1024, 128, "prefill"), (64, 4096, 768, 64, "prefill")])
def test_automatic_dispatch_at_its_edges(M, N, K, g, kernel):
    """Which kernel a plain call takes (they round differently: the one forced gives the same bits), and its result."""
    import quant
    lib = quant.load_library()
    p = packed(N, K, g)
    qw, zs = to_dev(p)
    x = make_x(M, K).cuda()
    auto = quant.gemm_awq_bias(x, qw, zs, None, N, g)
    forced = {}
    try:
        if M <= 64:
            lib.w4a16_tune_decode(3, 0, 0, 0)
            forced["batched"] = quant.gemm_awq_bias(x, qw, zs, None, N, g)
    finally:
        lib.w4a16_tune_decode(0, 0, 0, 0)
    forced["decode" if M <= 32 else "prefill"] = quant.gemm_awq_bias(x, qw, zs, None, N, g, algo=quant.ALGO_SKINNY if M <= 32 else quant.ALGO_TC)
    same = [k for k, v in forced.items() if torch.equal(v, auto)]
    assert same == [kernel], same
    if N * K <= 4096 * 2048:
        run(M, N, K, g, algo=0, bias=True)


@pytest.mark.parametrize("M,g", [(9, 64), (16, 64), (24, 128), (32, 128), (32, 64)])
def test_batched_decode_in_a_dependent_chain_of_static_weights(M, g):
    """The batched-decode kernel under programmatic launch (what a model's token step of 9 to 32 sequences runs): early weight
    copies, waits behind the previous grid, dependents launched early.  Every call consumes the previous one's output, with
    other kernels of the library in between; eagerly and replayed in a graph the bits are those of the plain launches."""
    import quant
    N = K = 1024
    devs = [to_dev(make_packed(N, K, g, seed=50 + i)) for i in range(3)]
    x = (make_x(M, K) * 0.5).cuda()
    weight = torch.ones(N, dtype=torch.float16, device="cuda")

    def chain(static):
        h = x
        for i in range(8):
            qw, zs = devs[i % 3]
            h = quant.gemm_awq_bias(h, qw, zs, None, N, g, static_weights=static, relu=i == 4, residual=h if i % 3 == 1 else None)
            if i % 3 == 2:
                h = quant.add_norm(h, None, weight, None, 1e-5, True)[1]
        return h

    plain = chain(False)
    assert bool(plain.isfinite().all()) and float(plain.float().abs().max()) > 0
    for _ in range(20):
        assert torch.equal(chain(True), plain)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain(True)
    for _ in range(20):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, plain)


@pytest.mark.parametrize("M,N,K,g", [(9, 416, 1344, 64), (24, 96, 1024, 128), (32, 1376, 512, 64), (40, 416, 2048, 128), (64, 32, 1024, 64)])
def test_batched_decode_relu(M, N, K, g):
    """ReLU and its order with bias and residual in the batched-decode kernel, also where the last block has few out-features."""
    import quant
    lib = quant.load_library()
    qw, zs = to_dev(packed(N, K, g))
    x = make_x(M, K).cuda()
    gen = torch.Generator().manual_seed(8)
    b, r = torch.randn(1, N, generator=gen).half().cuda(), torch.randn(1, M, N, generator=gen).half().cuda()
    try:
        lib.w4a16_tune_decode(3, 0, 0, 0)
        plain = quant.gemm_awq_bias(x, qw, zs, None, N, g)
        assert torch.equal(quant.gemm_awq_bias(x, qw, zs, None, N, g, relu=True), torch.relu(plain))
        assert torch.equal(quant.gemm_awq_bias(x, qw, zs, b, N, g, relu=True, residual=r), torch.relu(plain + b) + r)
    finally:
        lib.w4a16_tune_decode(0, 0, 0, 0)


def test_an_input_of_a_tensor_subclass_gives_a_plain_output():
    import quant

    class Tagged(torch.Tensor):
        pass

    N, K, g = 64, 256, 64
    qw, zs = to_dev(packed(N, K, g))
    x = make_x(3, K).cuda()
    plain = quant.gemm_awq_bias(x, qw, zs, None, N, g)
    for t in (x.as_subclass(Tagged), torch.nn.Parameter(x, requires_grad=False)):
        out = quant.gemm_awq_bias(t, qw, zs, None, N, g)
        assert type(out) is torch.Tensor and torch.equal(out, plain)
