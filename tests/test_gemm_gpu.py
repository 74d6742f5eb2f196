"""Numerics of the sm_100a GEMM kernel against a plain PyTorch fp32 reference."""
import os
import subprocess
import sys

import pytest
import torch

import flashoverlap_b200  # noqa: F401  (registers the classes)
from flashoverlap_b200.utils.config import ALGO_TILES

ALGOS = list(range(len(ALGO_TILES)))

pytestmark = pytest.mark.gpu


def _impl():
    impl = torch.classes.flashoverlap_class.OverlapImpl()
    impl.cutlass_init()
    impl.set_timeout_ms(2000)
    return impl


def _ref(A, B):
    return A.float() @ B.float().t()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("shape", [(128, 256, 64), (256, 512, 256), (512, 1024, 1000), (1024, 2048, 4096)])
def test_gemm_matches_fp32_reference(dtype, algo, shape):
    M, N, K = shape
    K = (K + 7) // 8 * 8
    if M % ALGO_TILES[algo][0] or N % ALGO_TILES[algo][1]:
        pytest.skip("shape is not a multiple of this tile")
    torch.manual_seed(0)
    A = torch.randn(M, K, device="cuda", dtype=dtype)
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).to(dtype)
    C = torch.full((M, N), float("nan"), device="cuda", dtype=dtype)
    impl = _impl()
    impl.set_keep_tile(True)     # this tile configuration and no other
    impl.cutlass_gemm(A, B, C, algo)
    torch.cuda.synchronize()
    impl.check_status()
    assert impl.last_algo() == algo
    ref = _ref(A, B)
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert torch.isfinite(C.float()).all(), "unwritten or non-finite output"
    err = (C.float() - ref).abs().max().item()
    assert err <= tol * max(1.0, ref.abs().max().item()), f"max abs err {err}"
    # and in the configuration that the launch chooses: the same sums in the same order
    D = torch.full_like(C, float("nan"))
    impl.set_keep_tile(False)
    impl.cutlass_gemm(A, B, D, algo)
    torch.cuda.synchronize()
    impl.check_status()
    assert impl.last_algo() == torch.ops.flashoverlap_op.planned_algo(M, N, K, algo, 0, False)
    assert torch.equal(C, D)


def test_gemm_many_tiles_persistent_loop():
    # more tiles than SMs: every CTA walks several tiles and both TMEM buffers
    M, N, K = 4096, 4096, 512
    torch.manual_seed(1)
    A = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).to(torch.bfloat16)
    C = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    impl = _impl()
    impl.set_keep_tile(True)
    for algo in ALGOS:
        C.fill_(float("nan"))
        impl.cutlass_gemm(A, B, C, algo)
        torch.cuda.synchronize()
        impl.check_status()
        assert impl.last_algo() == algo
        ref = _ref(A, B)
        err = (C.float() - ref).abs().max().item()
        assert err <= 2e-2 * ref.abs().max().item(), f"algo {algo}: max abs err {err}"


def test_gemm_repeated_calls_are_deterministic():
    M, N, K = 1024, 1024, 1024
    A = torch.randn(M, K, device="cuda", dtype=torch.float16)
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).half()
    impl = _impl()
    outs = []
    for _ in range(3):
        C = torch.empty(M, N, device="cuda", dtype=torch.float16)
        impl.cutlass_gemm(A, B, C, 0)
        outs.append(C)
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[1], outs[2])


def test_gemm_rejects_bad_shapes():
    impl = _impl()
    A = torch.randn(100, 64, device="cuda", dtype=torch.float16)
    B = torch.randn(256, 64, device="cuda", dtype=torch.float16)
    C = torch.empty(100, 256, device="cuda", dtype=torch.float16)
    with pytest.raises(RuntimeError):
        impl.cutlass_gemm(A, B, C, 0)
    with pytest.raises(RuntimeError):
        impl.cutlass_gemm(A.float(), B.float(), C.float(), 0)


def test_algo_table_matches_generated_python_copy():
    impl = _impl()
    assert impl.num_algos() == len(ALGO_TILES)
    assert [tuple(impl.algo_tile(a)) for a in ALGOS] == [tuple(t) for t in ALGO_TILES]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("algo,M,ffn", [(8, 256, 128), (3, 512, 1920), (9, 768, 64), (4, 256, 14336 // 8), (4, 256, 4800),
                                        (4, 256, 4864)])
@pytest.mark.parametrize("K", [8, 328])
@pytest.mark.parametrize("keep", [True, False])
def test_gemm_swiglu(dtype, algo, M, ffn, K, keep):
    # gate and up columns of one tile in the two CTAs of a pair, for each pair of at least 128 columns: one tile, many,
    # the narrowest; in the tile that the launch chooses also a last tile that is partly full (64 columns of 96, the last of
    # 4864)
    torch.manual_seed(ffn)
    impl = torch.classes.flashoverlap_class.OverlapImpl()
    impl.cutlass_init()
    impl.set_keep_tile(keep)
    x = torch.randn(M, K, device="cuda", dtype=dtype)
    w = (torch.randn(2 * ffn, K, device="cuda") * 2 / K ** 0.5).to(dtype)
    guard = torch.full((M + 1, ffn), 3.0, device="cuda", dtype=dtype)
    impl.gemm_swiglu(x, w, guard[:M], algo)
    torch.cuda.synchronize()
    assert impl.last_algo() == (algo if keep else torch.ops.flashoverlap_op.planned_algo(M, 2 * ffn, K, algo, 0, True))
    if (ffn, K, keep) == (4864, 328, False):
        half = torch.ops.flashoverlap_op.planned_tile(M, 2 * ffn, K, algo, 0, True, False)[1] // 2
        assert ffn % half == 64 and half > 64
    gate, up = (x.double() @ w.double().t()).chunk(2, dim=-1)
    want = torch.nn.functional.silu(gate) * up
    # one rounding of the result (11 or 8 bits) on fp32 sums
    eps = 2 ** -10.9 if dtype == torch.float16 else 2 ** -7.9
    assert ((guard[:M].double() - want).abs() <= eps * want.abs() + 1e-5).all()
    assert bool((guard[M] == 3).all())
    with pytest.raises(RuntimeError):
        impl.gemm_swiglu(x, w, guard[:M], 0)      # not a CTA-pair tile



@pytest.mark.parametrize("offset", [0, 8])
@pytest.mark.parametrize("algo,M,N", [(2, 128, 64), (7, 384, 192), (1, 128, 128), (0, 256, 768), (5, 256, 64), (8, 512, 2560)])
@pytest.mark.parametrize("glu", [False, True])
def test_gemm_result_on_16_and_32_byte_boundaries(offset, algo, M, N, glu):
    # eight warps share a tile's columns (one chunk of 32 each, an even and an odd number of them) and store 32 bytes at a
    # time where the result allows it, 16 elsewhere; the values around the result stay as they were
    if glu and (ALGO_TILES[algo][0] != 256 or ALGO_TILES[algo][1] < 128):
        pytest.skip("the gated form needs a pair tile of 128 columns")
    K = 72
    torch.manual_seed(N)
    A = torch.randn(M, K, device="cuda", dtype=torch.float16)
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).half()
    n = N // 2 if glu else N
    buf = torch.full((M * n + 32,), 5.0, device="cuda", dtype=torch.float16)
    C = buf[offset:offset + M * n].view(M, n)
    assert C.data_ptr() % 32 == 2 * offset
    impl = _impl()
    impl.set_keep_tile(True)
    (impl.gemm_swiglu if glu else impl.cutlass_gemm)(A, B, C, algo)
    torch.cuda.synchronize()
    impl.check_status()
    want = A.double() @ B.double().t()
    if glu:
        gate, up = want.chunk(2, dim=-1)
        want = torch.nn.functional.silu(gate) * up
    # one rounding to 11 bits of fp32 sums
    assert ((C.double() - want).abs() <= 2 ** -10.9 * want.abs() + 1e-5).all()
    assert bool((buf[:offset] == 5).all()) and bool((buf[offset + M * n:] == 5).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K,algo", [
    # K split over clusters of several sizes, some CTA without a column of its own, a last tile that is partly empty, K tails
    (128, 64, 4096, 2), (128, 1024, 28672, 2), (128, 1152, 20416, 1), (256, 1024, 15640, 1), (256, 1088, 8192, 2),
    (128, 2112, 6152, 2), (128, 10240, 8192, 6), (640, 640, 12296, 1),
    # tiles of 96, 160, 192 and 224 columns in pairs and single CTAs, one wave and several, last columns of all sorts
    (1152, 5120, 1720, 6), (3584, 2048, 4096, 8), (2048, 8192, 1024, 8), (1152, 1408, 2048, 6), (1024, 2560, 1128, 8),
    (896, 4672, 1040, 2)])
def test_gemm_in_tiles_of_any_width_and_split(dtype, M, N, K, algo):
    plan = torch.ops.flashoverlap_op.planned_tile(M, N, K, algo, 0, False, False)
    assert plan[3] > 1 or plan[1] < ALGO_TILES[plan[0]][1]      # a shape that is here for its plan
    torch.manual_seed(K)
    A = torch.randn(M, K, device="cuda", dtype=dtype)
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).to(dtype)
    impl = _impl()
    want = A.double() @ B.double().t()
    bits = 10.9 if dtype == torch.float16 else 7.9
    tiles = (M // ALGO_TILES[algo][0], N // ALGO_TILES[algo][1])
    count = tiles[0] * tiles[1]
    RA = torch.arange(count, dtype=torch.int32, device="cuda").flip(0).reshape(tiles)
    cseg = torch.tensor([count], dtype=torch.int32)
    MM = torch.zeros(tiles[0] + 1, tiles[1], dtype=torch.int32, device="cuda")
    over = torch.classes.flashoverlap_class.OverlapImpl()
    over.nccl_init(0, 1, [0] * 16)
    over.cutlass_init()
    over.overlap_init()
    over.set_timeout_ms(2000)
    first = None
    for offset in (0, 8, 0):
        buf = torch.full((M * N + 32,), 5.0, device="cuda", dtype=dtype)
        C = buf[offset:offset + M * N].view(M, N)
        impl.cutlass_gemm(A, B, C, algo)
        assert impl.last_algo() == plan[0]
        torch.cuda.synchronize()
        impl.check_status()
        # one rounding of fp32 sums
        assert ((C.double() - want).abs() <= 2 ** -bits * want.abs() + 4e-6 * K ** 0.5).all()
        assert bool((buf[:offset] == 5).all()) and bool((buf[offset + M * N:] == 5).all())
        assert first is None or torch.equal(C, first)          # the same bits every time
        first = C.clone()
    T = torch.full((M, N), float("nan"), device="cuda", dtype=dtype)
    over.gemm_allreduce_overlap(A, B, T, MM, RA, 1, cseg, cseg.cuda(), algo, False)
    torch.cuda.synchronize()
    over.check_status()
    from flashoverlap_b200.utils.reorder import from_tile_order
    assert torch.equal(from_tile_order(T, *ALGO_TILES[algo][:2], RA), first)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,N,K,algo", [(130, 1024, 4096, 1), (200, 2048, 4096, 2), (3, 1024, 28672, 2), (257, 1088, 8192, 2)])
def test_dispatch_of_ragged_rows_with_a_split_k(dtype, rows, N, K, algo):
    # rows that do not fill their tiles, few enough for the K of a tile to be split: the missing rows read as zero in every part
    impl = torch.classes.flashoverlap_class.OverlapImpl()
    impl.nccl_init(0, 1, [0] * 16)
    impl.cutlass_init()
    impl.set_timeout_ms(2000)
    mlen = torch.tensor([[rows]], dtype=torch.int32)
    padded = impl.a2a_padded_rows(mlen, algo)
    assert padded > rows and torch.ops.flashoverlap_op.planned_tile(padded, N, K, algo, 0, False, False)[3] > 1
    torch.manual_seed(rows)
    A = torch.randn(rows + 1, K, device="cuda").to(dtype)      # one row more than is sent
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).to(dtype)
    buf = torch.full((padded + 1, N), 5.0, device="cuda", dtype=dtype)
    impl.a2a_dispatch_gemm(A, B, buf[:padded], mlen, algo)
    torch.cuda.synchronize()
    impl.check_status()
    want = A[:rows].double() @ B.double().t()
    # one rounding of fp32 sums
    bits = 10.9 if dtype == torch.float16 else 7.9
    assert ((buf[:rows].double() - want).abs() <= 2 ** -bits * want.abs() + 4e-6 * K ** 0.5).all()
    assert bool((buf[padded:] == 5).all())


COOPERATIVE = """
import torch
import flashoverlap_b200
impl = torch.classes.flashoverlap_class.OverlapImpl()
impl.nccl_init(0, 1, [0] * 16)
impl.cutlass_init()
impl.set_timeout_ms(2000)
plan = torch.ops.flashoverlap_op.planned_tile
for M, N, K, algo, norm in [(128, 1024, 28672, 2, False), (640, 640, 12296, 1, False), (128, 8192, 1024, 7, True),
                            (256, 1664, 11904, 1, True), (2048, 2048, 256, 0, False)]:
    A = torch.randn(M, K, device="cuda", dtype=torch.float16)
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).half()
    want = A.double() @ B.double().t()
    if norm:
        C = impl.gemm_allreduce_fused(A, B, torch.ones(N, device="cuda", dtype=torch.float16), 1e-5, algo)
        want = want * torch.rsqrt(want.pow(2).mean(-1, keepdim=True) + 1e-5)
    else:
        C = torch.empty(M, N, device="cuda", dtype=torch.float16)
        impl.cutlass_gemm(A, B, C, algo)
    torch.cuda.synchronize()
    impl.check_status()
    # two roundings to 11 bits of fp32 sums over K
    assert ((C.double() - want).abs() <= 2 ** -9.9 * want.abs() + 1e-3).all(), (M, N, K)
    print("split", plan(M, N, K, algo, 0, False, norm)[3])
"""


def test_calls_with_the_cooperative_attribute():
    # every form of a launch, K split and not, where launches ask the driver for the residency of all CTAs
    env = dict(os.environ, FLASHOVERLAP_COOPERATIVE="1")
    res = subprocess.run([sys.executable, "-c", COOPERATIVE], env=env, capture_output=True, text=True, timeout=240,
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert res.returncode == 0, res.stderr[-2000:]
    assert "split 8" in res.stdout and "split 1" in res.stdout
