"""Every entry point of the reference's binding layer is registered, under the
CUDA names and under the names of the MUSA checkout (reference:
src/pybind.cpp:114-150), plus this library's fused entry points.  Runs without
a GPU: the classes can be constructed, only their methods need a device."""
import torch

import flashoverlap_b200  # noqa: F401  (loads the native library)

BASELINE = ["nccl_init", "cublas_init", "cublas_gemm", "nccl_allreduce", "nccl_reducescatter", "nccl_all2all",
            "mccl_init", "mublas_init", "mublas_gemm", "mccl_allreduce", "mccl_reducescatter", "mccl_all2all",
            "gemm_allreduce", "gemm_reducescatter", "gemm_all2all"]
OVERLAP_REFERENCE = ["cutlass_init", "nccl_init", "overlap_init", "cutlass_gemm", "mutlass_init", "mccl_init", "mutlass_gemm",
                     "gemm_allreduce_overlap", "gemm_reducescatter_overlap", "gemm_allreduce", "gemm_reducescatter",
                     "gemm_all2all", "nccl_allreduce", "nccl_reducescatter", "nccl_all2all", "mccl_allreduce",
                     "mccl_reducescatter", "mccl_all2all", "seg_allreduce"]
OVERLAP_OWN = ["gemm_allreduce_fused", "gemm_reducescatter_fused", "allgather_gemm", "a2a_dispatch_gemm", "a2a_padded_rows",
               "gemm_rmsnorm", "gemm_allreduce_twostream", "gemm_reducescatter_twostream", "set_timeout_ms", "set_sm_count",
               "set_raster_group", "set_raster_taper", "set_l2_hints", "set_use_nvls", "allreduce_uses_nvls",
               "set_allgather_multicast", "set_phase_trace", "set_row_trace", "status", "status_string", "check_status",
               "reset", "transport", "num_algos", "algo_tile", "p2p_push", "p2p_push_bulk", "multimem_bench",
               "detach_symmetric", "set_keep_tile", "last_algo", "gemm_swiglu"]
OPS = ["generate_nccl_id", "generate_mccl_id", "reorder_rmsnorm", "reorder_rmsnorm_eps", "rmsnorm", "add_rmsnorm", "tile_walk",
       "planned_algo"]


def test_baseline_class_has_the_reference_methods():
    obj = torch.classes.flashoverlap_class.BaselineImpl()
    missing = [m for m in BASELINE if not hasattr(obj, m)]
    assert not missing, missing


def test_overlap_class_has_the_reference_and_the_fused_methods():
    obj = torch.classes.flashoverlap_class.OverlapImpl()
    missing = [m for m in OVERLAP_REFERENCE + OVERLAP_OWN if not hasattr(obj, m)]
    assert not missing, missing


def test_ops_are_registered():
    missing = [o for o in OPS if not hasattr(torch.ops.flashoverlap_op, o)]
    assert not missing, missing
    ident = torch.ops.flashoverlap_op.generate_nccl_id()
    assert len(ident) == 16          # the reference's 128-byte id as 16 int64 (src/mccl_utils.cpp:7-14)


def test_planned_tile_needs_no_gpu():
    from flashoverlap_b200.utils.config import ALGO_TILES

    plan = torch.ops.flashoverlap_op.planned_algo
    for m, n, k in ((128, 64, 8), (1024, 2048, 4096), (4096, 8192, 8192), (16384, 14336, 28672)):
        for algo in range(len(ALGO_TILES)):
            assert 0 <= plan(m, n, k, algo, 148, False) < len(ALGO_TILES)
            assert ALGO_TILES[plan(m, n, k, algo, 1, False)][0] <= ALGO_TILES[algo][0]   # no pair on a single CTA
        bm, bn, _ = ALGO_TILES[plan(m, n, k, 8, 148, True)]
        assert bm == 256 and bn >= 128                                               # gate and up side by side


def test_planned_tile_is_not_one_that_measured_slower():
    # shapes at which the tile of the least single-wave time took 5 to 16 % longer than the named one (M, N, K, named)
    for m, n, k, algo in ((6656, 1024, 16232, 8), (3072, 2048, 792, 8), (1280, 640, 4424, 10), (4352, 1536, 10304, 8),
                          (2560, 2304, 6600, 8), (1024, 2560, 1128, 8), (768, 7168, 4056, 8), (3072, 2304, 5792, 8),
                          (6016, 8960, 440, 0), (1792, 1152, 2952, 4)):
        assert torch.ops.flashoverlap_op.planned_algo(m, n, k, algo, 148, False) == algo


def test_tile_table_matches_the_python_copy():
    from flashoverlap_b200.utils.config import ALGO_TILES

    obj = torch.classes.flashoverlap_class.OverlapImpl()
    assert obj.num_algos() == len(ALGO_TILES)
    for i, tile in enumerate(ALGO_TILES):
        assert tuple(obj.algo_tile(i))[:3] == tuple(tile)


def test_resident_plans_fit_the_chip():
    # every tile of a row block in one wave, whole chunks of 32 columns, tiles inside their configuration
    import random

    from flashoverlap_b200.utils.config import ALGO_TILES

    rng = random.Random(3)
    plan, seen = torch.ops.flashoverlap_op.planned_tile, 0
    for _ in range(400):
        ctas = rng.choice([1, 2, 37, 100, 148])
        algo = rng.randrange(len(ALGO_TILES))
        m, n = rng.randrange(1, 65) * ALGO_TILES[algo][0], rng.randrange(1, 40) * ALGO_TILES[algo][1]
        k = rng.randrange(1, 1024) * 8
        a, bn, rows, split, after = plan(m, n, k, algo, ctas, False, True)
        bm, width, _ = ALGO_TILES[a]
        assert after or split == 1
        if rows:
            seen += 1
            tiles = -(-n // bn)
            assert bn % 32 == 0 and 0 < bn <= width and 0 < rows <= -(-m // bm)
            assert rows * tiles * (bm // 128) <= ctas
        elif not after:
            assert bn == width
    assert seen > 100


def test_rmsnorm_kernel_behind_the_gemm_only_on_the_whole_chip():
    # a call that leaves SMs to other streams stays one kernel on the SMs it may use
    plan = torch.ops.flashoverlap_op.planned_tile
    for m, n, k, algo in [(256, 1664, 11904, 1), (128, 1024, 28672, 2), (384, 1280, 22256, 2), (2176, 4096, 4096, 0)]:
        assert plan(m, n, k, algo, 148, False, True)[4] == 1
        for ctas in (1, 2, 37, 100, 146, 147):
            assert list(plan(m, n, k, algo, ctas, False, True))[3:] == [1, 0]     # K in one piece, no second kernel


def test_plain_plans_fit_the_chip():
    # widths of whole chunks inside their configuration; a split over single CTAs that all run together, each with K to work
    # on; of the gated form two halves of whole chunks
    import random

    from flashoverlap_b200.utils.config import ALGO_TILES

    rng = random.Random(4)
    plan, narrow, splits = torch.ops.flashoverlap_op.planned_tile, 0, 0
    for i in range(600):
        ctas = rng.choice([1, 2, 37, 100, 148, 148, 148])
        glu = i % 4 == 0
        algo = rng.choice([3, 4, 8, 9]) if glu else rng.randrange(len(ALGO_TILES))
        m, n = rng.randrange(1, 17) * ALGO_TILES[algo][0], rng.randrange(1, 40) * ALGO_TILES[algo][1]
        k = rng.randrange(1, 3500) * 8
        a, bn, rows, split, after = plan(m, n, k, algo, ctas, glu, False)
        assert not after
        bm, width, bk = ALGO_TILES[a]
        assert rows == 0 and 0 < bn <= width and bn % (64 if glu else 32) == 0
        assert bm // 128 <= ctas or a == algo       # no pair on a single CTA that was not asked for
        assert not glu or (bm == 256 and bn >= 128)
        narrow += bn < width
        if split > 1:
            splits += 1
            assert not glu and bm == 128 and split <= 8
            assert -(-m // bm) * -(-n // bn) * split <= ctas and -(-k // bk) >= 3 * split
    assert narrow > 50 and splits > 30
