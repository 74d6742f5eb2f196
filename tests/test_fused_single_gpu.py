"""The fused kernel's reduce phase on one GPU (world size 1): GEMM + RMSNorm,
all-reduce / reduce-scatter entry points degenerate to a local reduction, the
reference-compatible reordered layout, the completion trace and RMSNorm ops.
Oracle: PyTorch fp32."""
import pytest
import torch

import flashoverlap_b200  # noqa: F401
from flashoverlap_b200.utils.config import ALGO_TILES
from flashoverlap_b200.utils.reorder import from_tile_order, reorder_indices, to_tile_order

pytestmark = pytest.mark.gpu


def rms_ref(x, w, eps):
    x = x.float()
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.float()


def make_impl():
    impl = torch.classes.flashoverlap_class.OverlapImpl()
    impl.nccl_init(0, 1, [0] * 16)
    impl.cutlass_init()
    impl.overlap_init()
    impl.set_timeout_ms(2000)
    return impl


def make_inputs(M, N, K, dtype, seed=0):
    torch.manual_seed(seed)
    A = torch.randn(M, K, device="cuda", dtype=dtype)
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).to(dtype)
    W = (1 + 0.1 * torch.randn(N, device="cuda")).to(dtype)
    return A, B, W


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("algo", list(range(len(ALGO_TILES))))
def test_gemm_rmsnorm_single_kernel(dtype, algo):
    M, N, K = 1024, 4096, 512
    A, B, W = make_inputs(M, N, K, dtype)
    C = torch.empty(M, N, device="cuda", dtype=dtype)
    O = torch.full((M, N), float("nan"), device="cuda", dtype=dtype)
    impl = make_impl()
    impl.set_keep_tile(True)     # this tile configuration and no other
    impl.gemm_rmsnorm(A, B, C, O, W, 1e-5, algo)
    torch.cuda.synchronize()
    impl.check_status()
    assert impl.last_algo() == algo
    ref = A.float() @ B.float().t()
    tol = 1e-2 if dtype == torch.float16 else 3e-2
    assert (C.float() - ref).abs().max().item() <= tol * ref.abs().max().item()
    want = rms_ref(C, W, 1e-5)  # the kernel normalises the 16-bit product it stored
    assert torch.isfinite(O.float()).all()
    assert (O.float() - want).abs().max().item() <= tol * want.abs().max().item()


@pytest.mark.parametrize("N", [512, 2304, 8192, 16384, 16640])
def test_gemm_rmsnorm_row_widths(N):
    # one unit of 512 columns per row (512), several with the last one half empty (2304), as many
    # weights as shared memory holds (8192), and rows whose weights come from memory (16384, 16640)
    M, K = 256, 128
    A, B, W = make_inputs(M, N, K, torch.float16, seed=N)
    C = torch.empty(M, N, device="cuda", dtype=torch.float16)
    O = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
    impl = make_impl()
    impl.gemm_rmsnorm(A, B, C, O, W, 1e-5, 0)
    torch.cuda.synchronize()
    impl.check_status()
    want = rms_ref(C, W, 1e-5)
    assert torch.isfinite(O.float()).all()
    assert (O.float() - want).abs().max().item() <= 1e-2 * want.abs().max().item()


def test_gemm_rmsnorm_more_rows_than_one_wave():
    # 8192 rows: every row group takes many units; the GEMM warps join the reduce phase
    M, N, K = 8192, 2048, 256
    A, B, W = make_inputs(M, N, K, torch.bfloat16, seed=21)
    C = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    O = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    impl = make_impl()
    for _ in range(2):
        impl.gemm_rmsnorm(A, B, C, O, W, 1e-5, 3)
    torch.cuda.synchronize()
    impl.check_status()
    want = rms_ref(C, W, 1e-5)
    assert torch.isfinite(O.float()).all()
    assert (O.float() - want).abs().max().item() <= 3e-2 * want.abs().max().item()


@pytest.mark.parametrize("algo,M,N", [(2, 128, 64), (2, 384, 4544), (7, 128, 8256), (5, 256, 1088), (8, 2816, 768)])
def test_norm_of_scattered_row_statistics(algo, M, N):
    # sums of squares from 1, 71, 129 and 17 tile columns (more than a lane loads at once), row ends inside a unit of 512
    # columns, weights beyond shared memory, more units than row groups; a plain call between two normalising ones
    # leaves the counters of the next call clean
    K = 200
    A, B, W = make_inputs(M, N, K, torch.float16, seed=N)
    impl = make_impl()
    y = (A.double() @ B.double().t())
    want = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * W.double()
    for norm in (True, False, True, True):
        out = impl.gemm_allreduce_fused(A, B, W if norm else None, 1e-5, algo)
        D = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
        impl.gemm_reducescatter_fused(A, B, D, W if norm else None, 1e-5, algo, False)
        torch.cuda.synchronize()
        impl.check_status()
        ref = want if norm else y
        # the product, its scaling and the weight are each rounded to 11 bits
        for got in (out, D):
            assert ((got.double() - ref).abs() <= 2 ** -9.3 * ref.abs() + 1e-4).all(), (norm, algo)


def test_norm_of_a_product_whose_staging_is_dropped():
    # 34 MB staged: its lines leave the L2 unwritten once they are read, and are written anew by the next calls
    M, N, K = 2048, 8256, 64
    impl = make_impl()
    for seed in range(3):
        A, B, W = make_inputs(M, N, K, torch.float16, seed=seed)
        out = impl.gemm_allreduce_fused(A, B, W, 1e-5, 5)
        D = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
        impl.gemm_reducescatter_fused(A, B, D, W, 1e-5, 5, False)
        torch.cuda.synchronize()
        impl.check_status()
        y = A.double() @ B.double().t()
        want = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * W.double()
        # the product, its scaling and the weight are each rounded to 11 bits
        for got in (out, D):
            assert ((got.double() - want).abs() <= 2 ** -9.3 * want.abs() + 1e-4).all()


def test_sms_left_to_another_stream_stay_free():
    # a GEMM on 100 SMs, then an RMSNorm that waits for it: the other SMs belong to whatever other streams bring meanwhile
    # (a CTA of this RMSNorm takes more than half of an SM's registers), and are not held by the waiting kernel
    M = N = K = 8192
    A, B, W = make_inputs(M, N, K, torch.bfloat16)
    impl = make_impl()
    impl.set_sm_count(100)
    C, O = torch.empty(M, N, device="cuda", dtype=torch.bfloat16), torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    x, y = A[:32].clone(), A[:32].clone()
    other = torch.cuda.Stream()
    waited = []
    for _ in range(4):
        start, end, mid = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        torch.cuda.synchronize()
        start.record()
        impl.cutlass_gemm(A, B, C, 8)
        torch.ops.flashoverlap_op.rmsnorm(C, O, W, 1e-5)
        end.record()
        with torch.cuda.stream(other):
            torch.ops.flashoverlap_op.rmsnorm(x, y, W, 1e-5)
            mid.record()
        torch.cuda.synchronize()
        waited.append(start.elapsed_time(mid) / start.elapsed_time(end))
    impl.check_status()
    assert sorted(waited)[1] < 0.5, waited


def test_phase_trace_records_every_row_once():
    M, N, K = 2048, 2048, 256
    A, B, W = make_inputs(M, N, K, torch.float16, seed=4)
    C = torch.empty(M, N, device="cuda", dtype=torch.float16)
    O = torch.empty(M, N, device="cuda", dtype=torch.float16)
    impl = make_impl()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    trace = torch.zeros(8 * sms, dtype=torch.int64, device="cuda")
    impl.set_phase_trace(trace)
    impl.gemm_rmsnorm(A, B, C, O, W, 1e-5, 0)
    torch.cuda.synchronize()
    impl.set_phase_trace(torch.empty(0, dtype=torch.int64, device="cuda"))
    t = trace.view(sms, 8).cpu()
    assert int(t[:, 5].sum()) == M            # rows reduced, over all CTAs
    assert int(t[:, 3].sum()) == (M // 128) * (N // 256)  # tiles computed
    assert bool((t[:, 1] >= t[:, 0]).all())   # GEMM phase ends after the start


@pytest.mark.parametrize("M,N,K,algo", [(128, 1024, 28672, 2), (256, 1088, 8192, 2), (640, 640, 12296, 1), (2048, 2048, 256, 0)])
def test_phase_trace_counts_every_tile_once(M, N, K, algo):
    # tiles of the named configuration, also where the launch splits their K over several CTAs
    A, B, _ = make_inputs(M, N, K, torch.float16)
    C = torch.empty(M, N, device="cuda", dtype=torch.float16)
    split = torch.ops.flashoverlap_op.planned_tile(M, N, K, algo, 0, False, False)[3]
    assert (split > 1) == (K > 256)
    impl = make_impl()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    trace = torch.zeros(8 * sms, dtype=torch.int64, device="cuda")
    impl.set_phase_trace(trace)
    impl.cutlass_gemm(A, B, C, algo)
    torch.cuda.synchronize()
    impl.set_phase_trace(torch.empty(0, dtype=torch.int64, device="cuda"))
    t = trace.view(sms, 8).cpu()
    assert int(t[:, 3].sum()) == (M // 128) * (N // ALGO_TILES[algo][1])     # pairs count 128 rows each
    assert bool((t[:, 1] >= t[:, 0]).all())


def test_row_trace_has_ordered_stamps_for_every_row():
    M, N, K = 1024, 2048, 256
    A, B, W = make_inputs(M, N, K, torch.float16, seed=5)
    C = torch.empty(M, N, device="cuda", dtype=torch.float16)
    O = torch.empty(M, N, device="cuda", dtype=torch.float16)
    impl = make_impl()
    rows = torch.zeros(6 * M, dtype=torch.int64, device="cuda")
    impl.set_row_trace(rows)
    impl.gemm_rmsnorm(A, B, C, O, W, 1e-5, 0)
    torch.cuda.synchronize()
    impl.set_row_trace(torch.empty(0, dtype=torch.int64, device="cuda"))
    impl.check_status()
    r = rows.view(6, M).cpu()
    claimed, stored, who, ready, summed, barrier = r[0], r[1], r[2], r[3], r[4], r[5]
    assert bool((claimed > 0).all())                       # every row was reduced by somebody
    assert bool((claimed <= ready).all() and (ready <= summed).all() and (summed <= barrier).all()
                and (barrier <= stored).all())
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert int(who.max()) < 4 * sms and int((who % 4).max()) <= 2   # CTA * 4 + row group (0..2)
    want = rms_ref(A.float() @ B.float().t(), W, 1e-5)
    assert (O.float() - want).abs().max().item() <= 1e-2 * want.abs().max().item()
    with pytest.raises(RuntimeError):
        impl.set_row_trace(torch.zeros(7, dtype=torch.int64, device="cuda"))  # not a multiple of 6
    # a buffer that is too small for the next call is ignored rather than overrun
    impl.set_row_trace(torch.zeros(6 * 128, dtype=torch.int64, device="cuda"))
    impl.gemm_rmsnorm(A, B, C, O, W, 1e-5, 0)
    torch.cuda.synchronize()
    impl.set_row_trace(torch.empty(0, dtype=torch.int64, device="cuda"))
    impl.check_status()


@pytest.mark.parametrize("with_norm", [False, True])
def test_world1_allreduce_and_reducescatter(with_norm):
    M, N, K = 512, 2048, 256
    A, B, W = make_inputs(M, N, K, torch.float16, seed=3)
    impl = make_impl()
    ref = A.float() @ B.float().t()
    want = rms_ref(ref, W, 1e-5) if with_norm else ref
    for _ in range(3):  # repeated calls alternate between the two buffer sets
        out = impl.gemm_allreduce_fused(A, B, W if with_norm else None, 1e-5, 0)
        torch.cuda.synchronize()
        impl.check_status()
        assert (out.float() - want).abs().max().item() <= 1e-2 * want.abs().max().item()
    D = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
    impl.gemm_reducescatter_fused(A, B, D, W if with_norm else None, 1e-5, 1, False)
    torch.cuda.synchronize()
    impl.check_status()
    assert (D.float() - want).abs().max().item() <= 1e-2 * want.abs().max().item()


@pytest.mark.parametrize("algo,M,N,K", [
    (2, 384, 2112, 4096), (1, 5504, 3456, 264), (6, 1152, 1408, 2048), (7, 128, 4672, 520), (0, 2432, 2816, 1000),
    (9, 2304, 8320, 136), (3, 256, 256, 64),
    # an odd number of 128-row blocks in pairs of them: the second half of the last tile row is empty; 256 columns, 128,
    # with a last tile column of 192 and of 64, and a staged product that is dropped
    (0, 2176, 4096, 4096), (0, 2432, 2816, 4096), (2, 384, 6336, 4096), (2, 640, 8256, 4096), (2, 1920, 8384, 2048)])
def test_gemm_in_another_tile_configuration(algo, M, N, K):
    # one rank: the named configuration says which shapes are accepted, the launch may take a larger tile whose last row
    # or column reaches past the matrix; natural order, tile order and RMSNorm
    A, B, W = make_inputs(M, N, K, torch.bfloat16, seed=K)
    impl = make_impl()
    y = A.double() @ B.double().t()
    guard = torch.full((M + 1, N), 7.0, device="cuda", dtype=torch.bfloat16)   # the row after the result
    C = guard[:M]
    impl.cutlass_gemm(A, B, C, algo)
    assert impl.last_algo() == torch.ops.flashoverlap_op.planned_algo(M, N, K, algo, 0, False)
    # the cases from 2176 rows on are here for their pair tiles: a planner that decides otherwise needs other shapes
    assert (ALGO_TILES[impl.last_algo()][0] == 256) == (K >= 2048 and N >= 2816)
    out = impl.gemm_allreduce_fused(A, B, W, 1e-5, algo)
    bm, bn, _ = impl.algo_tile(algo)
    tiles = (M // bm) * (N // bn)
    RA = reorder_indices(tiles, list(range(tiles))[::-1], device="cuda").reshape(M // bm, N // bn)
    cseg = torch.tensor([tiles], dtype=torch.int32)
    MM = torch.zeros((M // bm + 1, N // bn), dtype=torch.int32, device="cuda")
    T = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    impl.gemm_allreduce_overlap(A, B, T, MM, RA, 1, cseg, cseg.cuda(), algo, False)
    torch.cuda.synchronize()
    impl.check_status()
    top = y.abs().max().item()
    # rounding to 8 significant bits is off by at most 2^-8 of a value (and fp32 sums by far less); with RMSNorm three times
    assert (C.double() - y).abs().max().item() <= 1.01 * 2 ** -8 * top
    assert bool((guard[M] == 7).all())
    assert torch.equal(from_tile_order(T, bm, bn, RA), C)
    want = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * W.double()
    assert ((out.double() - want).abs() <= 2 ** -6.3 * want.abs() + 1e-4).all()


def test_compat_overlap_api_reordered_layout_and_trace():
    M, N, K, algo = 1024, 2048, 256, 0
    A, B, W = make_inputs(M, N, K, torch.float16, seed=5)
    impl = make_impl()
    bm, bn, _ = impl.algo_tile(algo)
    tm, tn = M // bm, N // bn
    tiles = tm * tn
    hint = [(7 * i + 3) % tiles for i in range(tiles)]  # a permutation since gcd(7, 64) = 1
    RA = reorder_indices(tiles, hint, device="cuda").reshape(tm, tn)
    cseg_cpu = torch.tensor([16, 16, 32], dtype=torch.int32)
    cseg_gpu = cseg_cpu.cuda()
    MM = torch.zeros((tm + 1, tn), dtype=torch.int32, device="cuda")
    C = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
    impl.gemm_allreduce_overlap(A, B, C, MM, RA, 1, cseg_cpu, cseg_gpu, algo, True)
    torch.cuda.synchronize()
    impl.check_status()
    ref = A.float() @ B.float().t()
    got = from_tile_order(C, bm, bn, RA)
    assert (got.float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item()
    # oracle for the layout itself
    assert torch.equal(to_tile_order(got, bm, bn, RA), C)
    flat = MM.flatten().cpu()
    assert int(flat[tn - 1]) == tiles  # ticket counter
    assert torch.equal(flat[tn:tn + tiles].sort().values, torch.arange(tiles, dtype=torch.int32))
    assert int(flat[:tn - 1].abs().sum()) == 0  # segment counters end at zero
    # reorder_rmsnorm undoes the layout
    out = torch.empty_like(C)
    torch.ops.flashoverlap_op.reorder_rmsnorm(C, out, W, bm, bn, 1, RA)
    torch.cuda.synchronize()
    want = rms_ref(got, W, 1e-5)
    assert (out.float() - want).abs().max().item() <= 1e-2 * want.abs().max().item()


@pytest.mark.parametrize("algo,rldn,keep", [(2, 1, False), (4, 2, False), (8, 1, False), (9, 4, False)] +
                         [(a, (1, 2, 4)[a % 3], True) for a in range(len(ALGO_TILES))])
@pytest.mark.parametrize("monitor", [False, True])
def test_compat_overlap_writes_tile_order_in_place(algo, rldn, keep, monitor):
    # one rank: the epilogue stores the tile-ordered result itself; tiles of every width, wide view rows, and a result
    # that takes the place of an operand (which then goes through the staging buffer)
    impl = make_impl()
    impl.set_keep_tile(keep)
    bm, bn, _ = impl.algo_tile(algo)
    M, N, K = 4 * bm, 8 * bn, 8 * bn
    A, B, _ = make_inputs(M, N, K, torch.bfloat16, seed=algo)
    RA = reorder_indices(32, [(11 * i + 5) % 32 for i in range(32)], device="cuda").reshape(4, 8)
    cseg = torch.tensor([20, 12], dtype=torch.int32)
    MM = torch.zeros((5, 8), dtype=torch.int32, device="cuda")
    C = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    impl.gemm_allreduce_overlap(A, B, C, MM, RA, rldn, cseg, cseg.cuda(), algo, monitor)
    assert impl.last_algo() == (algo if keep or monitor else torch.ops.flashoverlap_op.planned_algo(M, N, K, algo, 0, False))
    ref = A.double() @ B.double().t()
    want = to_tile_order(ref.to(torch.bfloat16), bm, bn, RA, rldn)
    torch.cuda.synchronize()
    impl.check_status()
    # one rounding to 8 bits
    assert (C.double() - want.double()).abs().max().item() <= 2 ** -7 * ref.abs().max().item()
    A2 = A.clone()
    MM.zero_()
    impl.gemm_allreduce_overlap(A2, B, A2, MM, RA, rldn, cseg, cseg.cuda(), algo, False)
    torch.cuda.synchronize()
    impl.check_status()
    assert torch.equal(A2, C) and impl.last_algo() == algo


@pytest.mark.parametrize("offset", [1, 3, 8])
def test_compat_overlap_result_at_any_element(offset):
    # a contiguous result that starts between two 16-byte boundaries (and one on a boundary)
    M, N, K, algo = 256, 512, 64, 0
    A, B, _ = make_inputs(M, N, K, torch.float16, seed=offset)
    impl = make_impl()
    bm, bn, _ = impl.algo_tile(algo)
    tm, tn = M // bm, N // bn
    RA = reorder_indices(tm * tn, [2, 0, 3, 1], device="cuda").reshape(tm, tn)
    cseg = torch.tensor([tm * tn], dtype=torch.int32)
    MM = torch.zeros((tm + 1, tn), dtype=torch.int32, device="cuda")
    want = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
    impl.gemm_allreduce_overlap(A, B, want, MM, RA, 1, cseg, cseg.cuda(), algo, False)
    buf = torch.full((M * N + 16,), 7.0, device="cuda", dtype=torch.float16)
    impl.gemm_allreduce_overlap(A, B, buf[offset:offset + M * N].view(M, N), MM, RA, 1, cseg, cseg.cuda(), algo, False)
    torch.cuda.synchronize()
    impl.check_status()
    assert torch.equal(buf[offset:offset + M * N].view(M, N), want)
    assert bool((buf[:offset] == 7).all()) and bool((buf[offset + M * N:] == 7).all())


def test_index_arrays_are_checked_anew_in_the_memory_of_an_earlier_one():
    # the outcome of a check belongs to the array, not to its address: a freed array's memory holds another one next
    M, N, K, algo = 256, 512, 64, 0
    A, B, W = make_inputs(M, N, K, torch.float16)
    impl = make_impl()
    C, O = (torch.empty(M, N, device="cuda", dtype=torch.float16) for _ in range(2))
    MM = torch.zeros((3, 2), dtype=torch.int32, device="cuda")
    cseg = torch.tensor([4], dtype=torch.int32)
    cseg_gpu = cseg.cuda()

    def overlap(ra):
        impl.gemm_allreduce_overlap(A, B, C, MM, ra, 1, cseg, cseg_gpu, algo, False)

    def norm(ra):
        torch.ops.flashoverlap_op.reorder_rmsnorm_eps(C, O, W, 128, 256, 1, ra, 1e-5)

    for call in (overlap, norm):
        good = torch.arange(4, dtype=torch.int32, device="cuda").view(2, 2)
        call(good)
        call(good)
        address = good.data_ptr()
        del good
        bad = torch.zeros(4, dtype=torch.int32, device="cuda").view(2, 2)     # one slot four times: in range, no order
        assert bad.data_ptr() == address
        with pytest.raises(RuntimeError, match="not a permutation"):
            call(bad)
        del bad
    torch.cuda.synchronize()
    impl.check_status()


def test_addresses_are_checked_on_the_host_before_any_launch():
    # the kernel moves 16 bytes at a time: whatever starts between two such boundaries is refused with a message
    M, N, K = 256, 512, 64
    A, B, W = make_inputs(M, N, K, torch.float16)
    impl = make_impl()

    def off(rows, cols):
        return torch.zeros(rows * cols + 8, device="cuda", dtype=torch.float16)[1:1 + rows * cols].view(rows, cols)

    C, O, w = torch.empty(M, N, device="cuda", dtype=torch.float16), off(M, N), off(1, N).view(N)
    half = torch.empty(M, N // 2, device="cuda", dtype=torch.float16)
    mlen = torch.tensor([[M]], dtype=torch.int32)
    bad = [
        lambda: impl.cutlass_gemm(A, B, O, 0),
        lambda: impl.gemm_swiglu(A, B, off(M, N // 2), 8),
        lambda: impl.gemm_rmsnorm(A, B, O, C, W, 1e-5, 0),
        lambda: impl.gemm_rmsnorm(A, B, C, O, W, 1e-5, 0),
        lambda: impl.gemm_rmsnorm(A, B, C, torch.empty_like(C), w, 1e-5, 0),
        lambda: impl.gemm_allreduce_fused(A, B, w, 1e-5, 0),
        lambda: impl.gemm_reducescatter_fused(A, B, O, None, 1e-5, 0, False),
        lambda: impl.gemm_reducescatter_fused(A, B, O, W, 1e-5, 0, False),
        lambda: impl.allgather_gemm(A, B, O, 0),
        lambda: impl.allgather_gemm(off(M, K), B, C, 0),
        lambda: impl.a2a_dispatch_gemm(A, B, O, mlen, 0),
        lambda: impl.a2a_dispatch_gemm(off(M, K), B, C, mlen, 0),
    ]
    for i, call in enumerate(bad):
        with pytest.raises(RuntimeError, match="16-byte aligned"):
            call()
            pytest.fail(f"call {i} was accepted")
    impl.gemm_swiglu(A, B, half, 8)                   # and nothing was broken on the way
    impl.allgather_gemm(A, B, C, 0)
    torch.cuda.synchronize()
    impl.check_status()
    assert (C.float() - A.float() @ B.float().t()).abs().max().item() < 0.1


def test_index_arrays_are_checked_on_the_host_before_any_launch():
    M, N, K, algo = 256, 512, 64, 0
    A, B, W = make_inputs(M, N, K, torch.float16)
    impl = make_impl()
    MM = torch.zeros((1, 2), dtype=torch.int32, device="cuda")
    C = torch.empty(M, N, device="cuda", dtype=torch.float16)
    cseg = torch.tensor([4], dtype=torch.int32)
    out_of_range = torch.tensor([[0, 1], [2, 400]], dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="outside"):
        impl.gemm_allreduce_overlap(A, B, C, MM, out_of_range, 1, cseg, cseg.cuda(), algo, False)
    duplicate = torch.tensor([[0, 1], [1, 3]], dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="permutation"):
        impl.gemm_allreduce_overlap(A, B, C, MM, duplicate, 1, cseg, cseg.cuda(), algo, False)
    with pytest.raises(RuntimeError, match="outside"):
        torch.ops.flashoverlap_op.reorder_rmsnorm(C, torch.empty_like(C), W, 128, 256, 1, out_of_range)
    # a tensor that passed the check is checked again after it has been written to
    RA = reorder_indices(4, [], device="cuda").reshape(2, 2)
    impl.gemm_allreduce_overlap(A, B, C, MM, RA, 1, cseg, cseg.cuda(), algo, False)
    RA[1, 1] = 77
    with pytest.raises(RuntimeError, match="outside"):
        impl.gemm_allreduce_overlap(A, B, C, MM, RA, 1, cseg, cseg.cuda(), algo, False)
    torch.cuda.synchronize()
    impl.check_status()


def test_compat_overlap_api_rejects_bad_segments():
    M, N, K, algo = 256, 512, 64, 0
    A, B, _ = make_inputs(M, N, K, torch.float16)
    impl = make_impl()
    RA = reorder_indices(4, [], device="cuda").reshape(2, 2)
    MM = torch.zeros((1, 2), dtype=torch.int32, device="cuda")
    C = torch.empty(M, N, device="cuda", dtype=torch.float16)
    bad = torch.tensor([1, 1], dtype=torch.int32)  # sums to 2, not 4: the reference would spin forever
    with pytest.raises(RuntimeError, match="sum"):
        impl.gemm_allreduce_overlap(A, B, C, MM, RA, 1, bad, bad.cuda(), algo, False)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dim", [512, 4096, 8192, 16384, 32768, 1000 * 8])
def test_rmsnorm_op(dtype, dim):
    torch.manual_seed(0)
    x = torch.randn(37, dim, device="cuda", dtype=dtype)
    w = (1 + 0.1 * torch.randn(dim, device="cuda")).to(dtype)
    o = torch.empty_like(x)
    torch.ops.flashoverlap_op.rmsnorm(x, o, w, 1e-6)
    torch.cuda.synchronize()
    want = rms_ref(x, w, 1e-6)
    tol = 1e-2 if dtype == torch.float16 else 3e-2
    assert (o.float() - want).abs().max().item() <= tol * want.abs().max().item()


@pytest.mark.parametrize("rows", [1, 296, 297, 2500])
@pytest.mark.parametrize("dim", [8, 256, 264, 8192, 8200, 16384, 16392, 32768, 32776])
def test_rmsnorm_thread_shapes(rows, dim):
    # one, two or four chunks per thread, a partly filled last warp, several rows per CTA, rows read twice; in place too
    torch.manual_seed(dim + rows)
    x = torch.randn(rows, dim, device="cuda", dtype=torch.float16)
    w = (1 + 0.1 * torch.randn(dim, device="cuda")).half()
    o = torch.full_like(x, float("nan"))
    torch.ops.flashoverlap_op.rmsnorm(x, o, w, 1e-6)
    xd = x.double()
    want = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    # two roundings to 11 bits each
    assert ((o.double() - want).abs() <= 2 ** -9.9 * want.abs() + 1e-7).all()
    torch.ops.flashoverlap_op.rmsnorm(x, x, w, 1e-6)
    assert torch.equal(x, o)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,dim", [(1481, 8200), (1500, 16384), (3000, 12296),      # four chunks per thread
                                      (12300, 5128), (10500, 6104), (7700, 8200), (3900, 16384)])     # 126 MB: a CTA per row
def test_rmsnorm_of_many_wide_rows(dtype, rows, dim):
    torch.manual_seed(dim)
    x = torch.randn(rows, dim, device="cuda", dtype=dtype)
    w = (1 + 0.1 * torch.randn(dim, device="cuda")).to(dtype)
    o = torch.full_like(x, float("nan"))
    torch.ops.flashoverlap_op.rmsnorm(x, o, w, 1e-6)
    xd = x.double()
    want = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    # two roundings to 11 or 8 bits each
    ulp = 2 ** -9.9 if dtype == torch.float16 else 2 ** -6.9
    assert ((o.double() - want).abs() <= ulp * want.abs() + 1e-7).all()
    torch.ops.flashoverlap_op.rmsnorm(x, x, w, 1e-6)
    assert torch.equal(x, o)


def test_rmsnorm_addresses_are_checked_on_the_host():
    op = torch.ops.flashoverlap_op
    rows, dim = 128, 256
    good = torch.ones(rows, dim, device="cuda", dtype=torch.float16)
    odd = torch.ones(rows * dim + 8, device="cuda", dtype=torch.float16)[3:3 + rows * dim].view(rows, dim)
    w, w_odd = good[0].clone(), odd[0]
    RA = torch.zeros(1, dtype=torch.int32, device="cuda")
    for x, o, g in ((odd, good, w), (good, odd, w), (good, good, w_odd)):
        for call in (lambda: op.rmsnorm(x, o, g, 1e-5), lambda: op.reorder_rmsnorm_eps(x, o, g, rows, dim, 1, RA, 1e-5),
                     lambda: op.add_rmsnorm(x, good, good, o, g, 1e-5)):
            with pytest.raises(RuntimeError, match="16-byte aligned"):
                call()


def test_rmsnorm_of_the_most_rows():
    # the row numbers of the last step of most CTAs lie past the largest int; in place, 34 GB
    rows = 2 ** 31 - 1
    if torch.cuda.mem_get_info()[0] < 40 * 2 ** 30:
        pytest.skip("needs 34 GB of device memory")
    x = torch.full((rows, 8), 3.0, device="cuda", dtype=torch.float16)
    w = torch.arange(1, 9, device="cuda", dtype=torch.float16)
    torch.ops.flashoverlap_op.rmsnorm(x, x, w, 1e-6)
    torch.cuda.synchronize()
    # equal values normalise to one (9 + 1e-6 rounds to 9 in fp32 up to one ulp, which fp16 does not see)
    for part in x.view(-1)[:rows // 16 * 128].view(16, -1, 8):
        assert torch.equal(part.amin(0), w) and torch.equal(part.amax(0), w)
    assert torch.equal(x[rows // 16 * 16:], w.expand(rows % 16, 8))
    del x, part
    torch.cuda.empty_cache()


@pytest.mark.parametrize("rows,dim", [(1, 8), (37, 8000), (600, 4096), (300, 16392), (3, 32776)])
def test_add_rmsnorm(rows, dim):
    torch.manual_seed(dim)
    x, r = torch.randn(2, rows, dim, device="cuda", dtype=torch.bfloat16)
    w = (1 + 0.1 * torch.randn(dim, device="cuda")).to(torch.bfloat16)
    s, o, o2 = (torch.full_like(x, float("nan")) for _ in range(3))
    torch.ops.flashoverlap_op.add_rmsnorm(x, r, s, o, w, 1e-5)
    torch.ops.flashoverlap_op.rmsnorm(x + r, o2, w, 1e-5)
    assert torch.equal(s, x + r) and torch.equal(o, o2)      # the two steps one after the other


def test_reorder_rmsnorm_rldn2():
    M, N, bm, bn = 512, 1024, 128, 256
    tm, tn = M // bm, N // bn
    torch.manual_seed(1)
    x = torch.randn(M, N, device="cuda", dtype=torch.float16)
    w = (1 + 0.1 * torch.randn(N, device="cuda")).half()
    RA = reorder_indices(tm * tn, [5, 1, 9, 0], device="cuda").reshape(tm, tn)
    for rldn in (1, 2, 4):
        xr = to_tile_order(x, bm, bn, RA, rldn)
        o = torch.empty_like(x)
        torch.ops.flashoverlap_op.reorder_rmsnorm(xr, o, w, bm, bn, rldn, RA)
        torch.cuda.synchronize()
        want = rms_ref(x, w, 1e-5)
        assert (o.float() - want).abs().max().item() <= 1e-2 * want.abs().max().item(), f"rldn={rldn}"


def test_allgather_gemm_world1():
    M, N, K = 512, 1024, 256
    A, B, _ = make_inputs(M, N, K, torch.bfloat16, seed=8)
    impl = make_impl()
    C = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    for algo in (0, 3):
        impl.allgather_gemm(A, B, C, algo)
        torch.cuda.synchronize()
        impl.check_status()
        ref = A.float() @ B.float().t()
        assert (C.float() - ref).abs().max().item() <= 3e-2 * ref.abs().max().item()


def test_a2a_dispatch_gemm_world1():
    K, N = 128, 256
    impl = make_impl()
    mlen = torch.tensor([[300]], dtype=torch.int32)
    A = torch.randn(300, K, device="cuda", dtype=torch.float16)
    B = (torch.randn(N, K, device="cuda") / K ** 0.5).half()
    m_pad = impl.a2a_padded_rows(mlen, 0)
    assert m_pad == 384
    C = torch.empty(m_pad, N, device="cuda", dtype=torch.float16)
    impl.a2a_dispatch_gemm(A, B, C, mlen, 0)
    torch.cuda.synchronize()
    impl.check_status()
    ref = A.float() @ B.float().t()
    assert (C[:300].float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item()
    with pytest.raises(RuntimeError):
        impl.a2a_dispatch_gemm(A[:100], B, C, mlen, 0)  # fewer rows than mLen says
    # whole tiles on one rank: the GEMM reads the caller's rows in place
    mlen2 = torch.tensor([[384]], dtype=torch.int32)
    A2 = torch.randn(384, K, device="cuda", dtype=torch.float16)
    C.fill_(float("nan"))
    impl.a2a_dispatch_gemm(A2, B, C, mlen2, 0)
    torch.cuda.synchronize()
    impl.check_status()
    ref2 = A2.float() @ B.float().t()
    assert (C.float() - ref2).abs().max().item() <= 1e-2 * ref2.abs().max().item()


@pytest.mark.parametrize("algo,rows,N,K", [(a, r, 512, 136) for a in (0, 8) for r in (1, 127, 129, 255, 257)] +
                         [(0, 2100, 4096, 4096), (1, 2427, 2816, 4096)])
def test_a2a_dispatch_gemm_ragged_rows_in_place(algo, rows, N, K):
    # rows that end inside the last tile: read where they are, the rest of the tile counts as zero; the last two cases in
    # pair tiles whose last second half holds nothing
    impl = make_impl()
    mlen = torch.tensor([[rows]], dtype=torch.int32)
    A, B, _ = make_inputs(rows, N, K, torch.float16, seed=rows)
    C = torch.full((impl.a2a_padded_rows(mlen, algo), N), float("nan"), device="cuda", dtype=torch.float16)
    impl.a2a_dispatch_gemm(A, B, C, mlen, algo)
    torch.cuda.synchronize()
    impl.check_status()
    assert rows < 2000 or ALGO_TILES[impl.last_algo()][0] == 256
    ref = A.double() @ B.double().t()
    # one rounding to 11 bits and fp32 sums
    assert (C[:rows].double() - ref).abs().max().item() <= 2 ** -10 * ref.abs().max().item()
    assert bool((C[rows:] == 0).all())


@pytest.mark.parametrize("rows,K,N", [(300, 512, 512), (1000, 1024, 256), (512, 256, 768)])
def test_a2a_dispatch_gemm_in_the_place_of_its_rows(rows, K, N):
    # the product overwrites the rows it is made of, from their first value on: narrower, as wide, wider than they are
    impl = make_impl()
    mlen = torch.tensor([[rows]], dtype=torch.int32)
    A, B, _ = make_inputs(rows, N, K, torch.float16, seed=K)
    m_pad = impl.a2a_padded_rows(mlen, 0)
    want = torch.empty((m_pad, N), device="cuda", dtype=torch.float16)
    impl.a2a_dispatch_gemm(A, B, want, mlen, 0)
    buf = torch.zeros(max(m_pad * N, rows * K), device="cuda", dtype=torch.float16)
    rows_view = buf[:rows * K].view(rows, K)
    rows_view.copy_(A)
    impl.a2a_dispatch_gemm(rows_view, B, buf[:m_pad * N].view(m_pad, N), mlen, 0)
    torch.cuda.synchronize()
    impl.check_status()
    assert torch.equal(buf[:rows * N].view(rows, N), want[:rows])


@pytest.mark.parametrize("heads,kv_heads", [(16, 16), (16, 4), (4, 2), (2, 1)])
def test_attention_of_grouped_heads_stores_no_scores(heads, kv_heads):
    # head widths 128 to 1024: one attention kernel each time, whose memory grows with the tokens and not their square
    from flashoverlap_b200.models.decoder_block import TPDecoderBlock

    hidden, batch, seq = 2048, 1, 2048
    block = TPDecoderBlock(make_impl(), hidden, 256, heads, kv_heads, 1e-5, 8, dtype=torch.bfloat16)
    hd = hidden // heads
    torch.manual_seed(heads)
    qkv = torch.randn(batch * seq, (heads + 2 * kv_heads) * hd, device="cuda", dtype=torch.bfloat16)
    block._attention(qkv, batch, seq)                   # whatever the first call keeps
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    got = block._attention(qkv, batch, seq)
    used = torch.cuda.max_memory_allocated() - before
    # the output, its copy, repeated keys and values, each as large as the queries, and as much again for padding
    assert used <= 8 * batch * seq * hidden * 2, f"{used >> 20} MB"
    q, k, v = (z.reshape(batch, seq, -1, hd).transpose(1, 2).double()
               for z in qkv.split([hidden, kv_heads * hd, kv_heads * hd], dim=-1))
    k, v = (z.repeat_interleave(heads // kv_heads, dim=1) for z in (k, v))
    mask = torch.ones(seq, seq, dtype=torch.bool, device="cuda").triu(1)
    want = (q @ k.transpose(-1, -2) / hd ** 0.5).masked_fill(mask, float("-inf")).softmax(-1) @ v
    want = want.transpose(1, 2).reshape(batch * seq, hidden)
    # probabilities and results are rounded to 8 bits: each within 2^-8 of values up to the largest one
    assert (got.double() - want).abs().max().item() <= 2 ** -7 * want.abs().max().item()


def test_host_feeder_double_buffers_inputs():
    from flashoverlap_b200.utils.pipeline import HostFeeder

    feeder = HostFeeder((64, 32), torch.float16)
    batches = [torch.full((64, 32), float(i), dtype=torch.float16).pin_memory() for i in range(5)]
    feeder.submit(batches[0])
    seen = []
    for i in range(1, 6):
        x = feeder.take()
        if i < 5:
            feeder.submit(batches[i])
        y = x.float().mean()  # stands for the step's compute
        feeder.release(x)
        seen.append(y)
    torch.cuda.synchronize()
    assert [float(v) for v in seen] == [0.0, 1.0, 2.0, 3.0, 4.0]


RESIDENT = [
    # M, N, K, named configuration, plan (configuration, tile columns, tile rows per wave)
    (128, 64, 64, 2, (7, 32, 1)),           # the narrowest tiles: the second half of the columns is empty
    (128, 8192, 1024, 7, (6, 128, 1)),      # one row block over 64 CTAs: statistics in more than one batch
    (384, 4544, 200, 2, (6, 128, 3)),       # the last tile column holds 64
    (2048, 8256, 64, 5, (0, 224, 4)),       # four waves, seven chunks of columns for two warps
    (1152, 5120, 1720, 1, (8, 224, 3)),     # pairs, the second half of the last tile row is empty; two waves
    (4096, 8192, 1024, 8, (8, 224, 2)),     # every SM, eight waves
    (2048, 4096, 2048, 8, (8, 256, 4)),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K,algo,plan", RESIDENT)
def test_resident_norm_matches_the_staged_form(dtype, M, N, K, algo, plan):
    # rows that stay on the chip between the product and its RMSNorm, call after call with another shape in between (the
    # exchange has to be left clean), results on a 32-byte boundary and on a 16-byte one; the same call with the named tile
    # kept goes through the staging buffer
    assert tuple(torch.ops.flashoverlap_op.planned_tile(M, N, K, algo, 0, False, True))[:3] == plan
    A, B, W = make_inputs(M, N, K, dtype, seed=N)
    A2, B2, W2 = make_inputs(256, 1024, 264, dtype, seed=1)
    impl = make_impl()
    y = A.double() @ B.double().t()
    want = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * W.double()
    y2 = A2.double() @ B2.double().t()
    want2 = y2 * torch.rsqrt(y2.pow(2).mean(-1, keepdim=True) + 1e-5) * W2.double()
    # the product, its scaling and the weight are each rounded to 11 or 8 bits
    rel = 2 ** -9.3 if dtype == torch.float16 else 2 ** -6.3
    buf = torch.empty(M * N + 32, device="cuda", dtype=dtype)
    first = None
    for offset in (0, 8, 0):
        buf.fill_(9.0)
        D = buf[offset:offset + M * N].view(M, N)
        impl.gemm_reducescatter_fused(A, B, D, W, 1e-5, algo, False)
        assert impl.last_algo() == plan[0]
        small = impl.gemm_allreduce_fused(A2, B2, W2, 1e-5, 2)
        torch.cuda.synchronize()
        impl.check_status()
        assert ((D.double() - want).abs() <= rel * want.abs() + 1e-4).all()
        assert ((small.double() - want2).abs() <= rel * want2.abs() + 1e-4).all()
        assert bool((buf[:offset] == 9).all()) and bool((buf[offset + M * N:] == 9).all())
        assert first is None or torch.equal(D, first)      # the same bits every time
        first = D.clone()
    impl.set_keep_tile(True)
    out = impl.gemm_allreduce_fused(A, B, W, 1e-5, algo)
    torch.cuda.synchronize()
    impl.check_status()
    assert impl.last_algo() == algo
    assert ((out.double() - want).abs() <= rel * want.abs() + 1e-4).all()


def test_resident_norm_in_a_graph():
    # replays run with the parameters of the capture: what one replay leaves in the exchange would be taken for the next
    # one's statistics
    M, N, K = 384, 4544, 200
    A, B, W = make_inputs(M, N, K, torch.float16)
    impl = make_impl()
    D = torch.empty(M, N, device="cuda", dtype=torch.float16)
    E = torch.empty_like(D)

    def calls():
        impl.gemm_reducescatter_fused(A, B, D, W, 1e-5, 2, False)      # RMSNorm: resident
        impl.gemm_reducescatter_fused(A, B, E, None, 1e-5, 2, False)   # none (an even number of fused calls)

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        calls()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        calls()
    for seed in range(3):
        A2, _, _ = make_inputs(M, N, K, torch.float16, seed=10 + seed)
        A.copy_(A2 * (seed + 1))
        graph.replay()
        torch.cuda.synchronize()
        impl.check_status()
        y = A.double() @ B.double().t()
        want = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * W.double()
        # the product, its scaling and the weight are each rounded to 11 bits
        assert ((D.double() - want).abs() <= 2 ** -9.3 * want.abs() + 1e-4).all()
        assert ((E.double() - y).abs() <= 2 ** -10.9 * y.abs() + 1e-5).all()


@pytest.mark.parametrize("operand,norm", [("A", False), ("A", True), ("B", False)])
def test_reducescatter_into_an_operand(operand, norm):
    # a result that takes the place of the rows (or, without RMSNorm, of the weights) that the GEMM reads while it stores tiles
    M = N = K = 2048
    A, B, W = make_inputs(M, N, K, torch.float16)
    impl = make_impl()
    want = torch.empty(M, N, device="cuda", dtype=torch.float16)
    weight = W if norm else None
    impl.gemm_reducescatter_fused(A, B, want, weight, 1e-5, 3, False)
    X, Y = A.clone(), B.clone()
    D = X if operand == "A" else Y
    impl.gemm_reducescatter_fused(X, Y, D, weight, 1e-5, 3, False)
    torch.cuda.synchronize()
    impl.check_status()
    assert torch.equal(D, want)


def test_resident_norm_of_rows_that_are_not_finite():
    # a sum of squares that is infinite or not a number passes the exchange like any other, and stays in its row; the next call
    # finds the exchange clean
    M, N, K = 384, 4544, 200
    assert torch.ops.flashoverlap_op.planned_tile(M, N, K, 2, 0, False, True)[2] > 0
    A, B, W = make_inputs(M, N, K, torch.float16)
    impl = make_impl()
    clean = impl.gemm_allreduce_fused(A, B, W, 1e-5, 2).clone()
    bad = {5: float("nan"), 130: float("inf"), 383: float("-inf"), 200: 60000.0, 201: 0.0}
    A2 = A.clone()
    for row, value in bad.items():
        A2[row] = value
    got = impl.gemm_allreduce_fused(A2, B, W, 1e-5, 2).clone()
    again = impl.gemm_allreduce_fused(A, B, W, 1e-5, 2).clone()
    torch.cuda.synchronize()
    impl.check_status()
    y = (A2.float() @ B.float().t()).half().float()       # as the 16-bit product holds it
    want = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * W.float()
    rest = torch.ones(M, dtype=torch.bool, device="cuda")
    rest[list(bad)] = False
    assert torch.equal(got[rest], clean[rest]) and torch.equal(again, clean)
    assert bool(got[5].isnan().all()) and bool((got[201] == 0).all())
    for row in (130, 200, 383):
        # infinities of the product times a scale of zero, zeros (or a finite row's values) elsewhere
        assert torch.equal(got[row].isnan(), want[row].isnan()), row
        fine = ~want[row].isnan()
        # a value of the product may round the other way (one unit of 11 bits), then two roundings
        assert ((got[row][fine].float() - want[row][fine]).abs() <= 2 ** -9 * want[row][fine].abs() + 1e-4).all()


@pytest.mark.parametrize("M,N,K,algo", [(256, 1664, 11904, 1), (2176, 4096, 4096, 0)])
@pytest.mark.parametrize("sms", [2, 37, 100])
def test_norm_on_some_of_the_sms(M, N, K, algo, sms):
    # shapes whose RMSNorm is a kernel behind the GEMM on the whole chip: on some of its SMs they stay one kernel
    plan = torch.ops.flashoverlap_op.planned_tile
    assert plan(M, N, K, algo, 0, False, True)[4] == 1 and plan(M, N, K, algo, sms, False, True)[4] == 0
    A, B, W = make_inputs(M, N, K, torch.bfloat16, seed=N)
    impl = make_impl()
    impl.set_sm_count(sms)
    want = norm_oracle(A, B, W)
    for _ in range(2):
        out = impl.gemm_allreduce_fused(A, B, W, 1e-5, algo)
        torch.cuda.synchronize()
        impl.check_status()
        assert impl.last_algo() == plan(M, N, K, algo, sms, False, True)[0]
        assert ((out.double() - want).abs() <= 2 ** -6.3 * want.abs() + 1e-4).all()   # three roundings to 8 bits


def norm_oracle(A, B, W):
    y = A.double() @ B.double().t()
    return y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * W.double()


def small_resident_call(impl):
    M, N, K = 128, 8192, 1024
    assert torch.ops.flashoverlap_op.planned_tile(M, N, K, 7, 0, False, True)[2] == 1
    A, B, W = make_inputs(M, N, K, torch.float16)
    out = impl.gemm_allreduce_fused(A, B, W, 1e-5, 7)
    torch.cuda.synchronize()
    impl.check_status()
    want = norm_oracle(A, B, W)
    assert ((out.double() - want).abs() <= 2 ** -9.3 * want.abs() + 1e-4).all()   # three roundings to 11 bits


def test_resident_norm_while_the_workspace_grows():
    # the exchange of row statistics is part of the workspace: it moves with it and starts clean
    impl = make_impl()
    small_resident_call(impl)
    for M, N, K in [(384, 4544, 200), (2048, 4096, 2048), (256, 1024, 264), (4096, 8192, 1024)]:
        A, B, W = make_inputs(M, N, K, torch.float16, seed=M)
        D = torch.empty(M, N, device="cuda", dtype=torch.float16)
        impl.gemm_reducescatter_fused(A, B, D, W, 1e-5, 2, False)
        torch.cuda.synchronize()
        want = norm_oracle(A, B, W)
        assert ((D.double() - want).abs() <= 2 ** -9.3 * want.abs() + 1e-4).all()
        small_resident_call(impl)


def test_workspace_that_cannot_grow_or_be_attached():
    # an allocation that fails leaves an engine that works: room for the four buffers of a 16384 x 16384 problem, but for
    # little more; then memory that is refused because it is too small
    impl = make_impl()
    small_resident_call(impl)
    M = N = 16384
    A, B, W = make_inputs(M, N, 8, torch.float16)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    spare = 8 * M * N + (16 << 20)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - spare, dtype=torch.uint8, device="cuda")
    with pytest.raises(RuntimeError, match="cudaMalloc"):
        impl.gemm_allreduce_fused(A, B, W, 1e-5, 8)
    del hold
    torch.cuda.empty_cache()
    small_resident_call(impl)
    tiny = torch.empty(1 << 18, dtype=torch.uint8, device="cuda")
    with pytest.raises(RuntimeError, match="too small"):
        impl.attach_symmetric([tiny.data_ptr()], 0, tiny.numel())
    small_resident_call(impl)


def test_resident_norm_in_attached_memory():
    # as large as the two products that the workspace is asked for: every call is accepted, also where the exchange has no room
    M, N, K = 4096, 8192, 256
    impl = make_impl()
    buf = torch.empty(8 * M * N + (4 << 20), dtype=torch.uint8, device="cuda")
    base = (buf.data_ptr() + 1023) // 1024 * 1024
    impl.attach_symmetric([base], 0, buf.numel() - 1024)
    A, B, W = make_inputs(M, N, K, torch.float16)
    for _ in range(2):
        out = impl.gemm_allreduce_fused(A, B, W, 1e-5, 8)
        torch.cuda.synchronize()
        impl.check_status()
        want = norm_oracle(A, B, W)
        assert ((out.double() - want).abs() <= 2 ** -9.3 * want.abs() + 1e-4).all()
        small_resident_call(impl)
    impl.detach_symmetric()
    small_resident_call(impl)


def test_wrappers_that_make_their_result_natively():
    # the same bits as the forms that write into a given tensor, rows of any count, and the same refusals
    M, N, K, algo = 300, 512, 136, 8
    A, B, W = make_inputs(M, N, K, torch.float16)
    impl = make_impl()
    from flashoverlap_b200 import ops

    x = torch.randn(37, 520, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(520, device="cuda", dtype=torch.bfloat16)
    out = torch.empty_like(x)
    torch.ops.flashoverlap_op.rmsnorm(x, out, w, 1e-5)
    assert torch.equal(ops.rmsnorm(x, w), out)
    RA = torch.arange(8, dtype=torch.int32, device="cuda").flip(0).reshape(2, 4)
    y = torch.randn(256, 512, device="cuda", dtype=torch.float16)
    out = torch.empty_like(y)
    torch.ops.flashoverlap_op.reorder_rmsnorm_eps(y, out, W, 128, 128, 2, RA, 1e-5)
    assert torch.equal(ops.reorder_rmsnorm(y, W, 128, 128, RA, 2), out)
    mlen = torch.tensor([[M]], dtype=torch.int32)
    C = torch.empty(512, N, device="cuda", dtype=torch.float16)
    impl.a2a_dispatch_gemm(A, B, C, mlen, algo)
    got = ops.a2a_dispatch_gemm(impl, A, B, mlen, 0, algo)
    assert got.shape == (M, N) and torch.equal(got, C[:M])
    assert torch.equal(ops.a2a_dispatch_gemm(impl, A, B, mlen, -1, algo), C[:M])
    assert ops.a2a_dispatch_gemm(impl, A, B, torch.tensor([[0]], dtype=torch.int32), 0, algo).shape == (0, N)
    for bad in (lambda: ops.rmsnorm(x[:, ::2], w[:260]), lambda: ops.rmsnorm(x, w[:512]), lambda: ops.rmsnorm(x.float(), w),
                lambda: ops.reorder_rmsnorm(y, W, 96, 128, RA, 2), lambda: ops.a2a_dispatch_gemm(impl, A, B, mlen + 1, 0, algo),
                lambda: ops.a2a_dispatch_gemm(impl, A, B, mlen, 1, algo)):
        with pytest.raises(RuntimeError):
            bad()
    torch.cuda.synchronize()
    impl.check_status()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,N,K,algo", [(256, 1664, 11904, 1), (128, 1024, 28672, 2), (384, 1280, 22256, 2), (2176, 4096, 4096, 0)])
def test_norm_behind_a_plain_gemm(dtype, M, N, K, algo):
    # few tiles and a long K: a GEMM whose K is split, then the RMSNorm kernel; also where a plain GEMM has the better tiles;
    # a call without RMSNorm and a resident one in between
    plan = torch.ops.flashoverlap_op.planned_tile(M, N, K, algo, 0, False, True)
    assert plan[4] == 1 and plan[2] == 0
    A, B, W = make_inputs(M, N, K, dtype, seed=N)
    impl = make_impl()
    y = A.double() @ B.double().t()
    want = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * W.double()
    # the product, its scaling and the weight are each rounded to 11 or 8 bits
    rel = 2 ** -9.3 if dtype == torch.float16 else 2 ** -6.3
    first = None
    for offset in (0, 8):
        buf = torch.full((M * N + 32,), 9.0, device="cuda", dtype=dtype)
        D = buf[offset:offset + M * N].view(M, N)
        impl.gemm_reducescatter_fused(A, B, D, W, 1e-5, algo, False)
        assert impl.last_algo() == plan[0]
        out = impl.gemm_allreduce_fused(A, B, W, 1e-5, algo)
        plain = impl.gemm_allreduce_fused(A[:, :264].contiguous(), B[:, :264].contiguous(), None, 1e-5, algo)
        torch.cuda.synchronize()
        impl.check_status()
        assert torch.isfinite(plain.float()).all()
        for got in (D, out):
            assert ((got.double() - want).abs() <= rel * want.abs() + 1e-4).all()
        assert bool((buf[:offset] == 9).all()) and bool((buf[offset + M * N:] == 9).all())
        assert first is None or torch.equal(D, first)
        first = D.clone()
