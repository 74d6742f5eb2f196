"""The tuning pipeline end to end on one GPU (world size 1): tile profiling,
bandwidth-curve file, completion-order hint, predictive and exhaustive search,
stage-2 file consumed by the reference-compatible layer."""
import pytest
import torch

import flashoverlap_b200  # noqa: F401
from flashoverlap_b200.models import OverlapRowParallelLayer, ReorderRMSNorm
from flashoverlap_b200.parallel import make_overlap_impl
from flashoverlap_b200.tune import search
from flashoverlap_b200.tune.runtime import compute_hint, measure_row_us, perf_running, profile_gemm
from flashoverlap_b200.utils import config as cfg

pytestmark = pytest.mark.gpu


def tiles_of(data, M, N):
    return (M // data["BM"]) * (N // data["BN"])


def test_profile_hint_search_and_use(tmp_path):
    M, N, K = 1024, 2048, 256
    impl = make_overlap_impl(timeout_ms=3000)
    BM, BN, dur, algo = profile_gemm(impl, M, N, K, torch.float16, warmup=2, reps=5)
    assert len(algo) == min(10, len(cfg.ALGO_TILES)) and dur == sorted(dur) and all(d > 0 for d in dur)
    cfg.save_stage1(M, N, K, BM, BN, dur, algo, tmp_path)

    tiles = (M // BM[0]) * (N // BN[0])
    ok, hint = compute_hint(impl, M, N, K, BM[0], BN[0], algo[0], 148 // (BM[0] // 128), "all_reduce",
                            warmup=2, samples=6)
    assert ok and sorted(hint) == list(range(tiles))

    curve = torch.tensor([[2.0 ** 20, 200.0], [2.0 ** 26, 400.0]])
    cfg.save_bandwidth(curve, "all_reduce", 1, path=tmp_path)
    sol = search.predictive_search(impl, M, N, K, "all_reduce", cfg.load_bandwidth("all_reduce", 1, path=tmp_path),
                                   path=tmp_path, reps=5, verbose=False)
    data = cfg.load_config(M, N, K, tmp_path)
    cfg.validate_stage2(data, M, N)
    assert data["Algo"] == sol["Algo"] and data["search"] == "predictive" and data["fused_dur"] > 0
    assert sum(data["cSeg"]) == tiles_of(data, M, N) and data["two_stream_dur"] > 0 and data["candidates_timed"] >= 1

    # exhaustive search on the same stage-1 lists: every candidate is timed, the file is rewritten
    ex = search.exhaustive_search(impl, M, N, K, "all_reduce", path=tmp_path, reps=3, verbose=False, seg_reps=3)
    data = cfg.load_config(M, N, K, tmp_path)
    cfg.validate_stage2(data, M, N)
    assert data["search"] == "exhaustive" and data["Algo"] == ex["Algo"]

    # the tuned file drives the reference-compatible layer + reorder-aware RMSNorm
    layer = OverlapRowParallelLayer(0, 1, K, N, M, data, "all_reduce", [0] * 16)
    norm = ReorderRMSNorm(N, M, data["BM"], data["BN"], data["hint"], eps=1e-5)
    with torch.no_grad():
        layer.weight.normal_(0.0, 1.0 / K ** 0.5)
        norm.weight.fill_(1.0)
        x = torch.randn(M, K, device="cuda", dtype=torch.float16)
        y = norm(layer(x))
    torch.cuda.synchronize()
    layer.overlap_class.check_status()
    ref = x.float() @ layer.weight.float().t()
    ref = ref * torch.rsqrt(ref.pow(2).mean(-1, keepdim=True) + 1e-5)
    assert (y.float() - ref).abs().max().item() < 2e-2
    impl.check_status()


class Recorder:
    """Passes calls on to an OverlapImpl and notes, for those that launch the kernel, which tile configuration was named
    (the position of the argument) and which one ran."""
    NAMED = {"cutlass_gemm": 3, "gemm_allreduce_fused": 4, "gemm_reducescatter_fused": 5, "gemm_allreduce_overlap": 8,
             "gemm_reducescatter_overlap": 10, "gemm_allreduce": 3, "gemm_reducescatter": 4}

    def __init__(self, impl):
        self.impl, self.ran = impl, []

    def __getattr__(self, name):
        method = getattr(self.impl, name)
        if name not in self.NAMED:
            return method

        def call(*args):
            out = method(*args)
            self.ran.append((name, args[self.NAMED[name]], self.impl.last_algo()))
            return out
        return call


def test_searches_time_the_tile_they_name():
    # on one rank a plain call runs the configuration with the least expected time, whatever it names; a search must not
    M, N, K = 1024, 2048, 4096
    impl = make_overlap_impl(timeout_ms=3000)
    rec = Recorder(impl)
    profile_gemm(rec, M, N, K, torch.float16, warmup=1, reps=2, rasters=(0, 2))
    for op in ("all_reduce", "reduce_scatter"):
        measure_row_us(rec, 2048, op, torch.float16, algo=4, M=1024, warmup=1, reps=1)
        for cseg in ([63, 1], [64]):
            perf_running(rec, M, N, K, 128, 256, 0, cseg, [], op, warmup=1, reps=1, raster_group=0)
    assert {a for name, a, _ in rec.ran if name == "cutlass_gemm"} == set(range(len(cfg.ALGO_TILES)))
    assert {name for name, _, _ in rec.ran} == set(Recorder.NAMED)
    assert all(asked == ran for _, asked, ran in rec.ran), rec.ran
    # and afterwards the launch chooses again
    A = torch.randn(M, K, device="cuda", dtype=torch.float16)
    B = torch.randn(N, K, device="cuda", dtype=torch.float16)
    C = torch.empty(M, N, device="cuda", dtype=torch.float16)
    planned = [torch.ops.flashoverlap_op.planned_algo(M, N, K, a, 0, False) for a in range(len(cfg.ALGO_TILES))]
    for a, p in enumerate(planned):
        impl.cutlass_gemm(A, B, C, a)
        assert impl.last_algo() == p
    assert planned != list(range(len(cfg.ALGO_TILES)))
    torch.cuda.synchronize()
    impl.check_status()


def test_layers_run_a_searched_configuration_as_named():
    from flashoverlap_b200.models import FusedRowParallelLinear

    M, N, K, algo = 1024, 2048, 4096, 5
    chosen = torch.ops.flashoverlap_op.planned_algo(M, N, K, algo, 0, False)
    assert chosen != algo        # a shape at which one rank would take another tile
    x = torch.randn(M, K, device="cuda", dtype=torch.float16) / K ** 0.5
    impl = make_overlap_impl(timeout_ms=3000)
    outs = []
    for op in ("all_reduce", "reduce_scatter"):
        for norm in (False, True):
            for config, ran in (({"Algo": algo, "raster_group": 4, "comm_op": op}, algo),
                                ({"Algo": algo, "comm_op": op}, chosen)):     # no raster group: not from this search
                torch.manual_seed(1)
                layer = FusedRowParallelLinear.from_config(impl, config, K, N, norm=norm)
                outs.append(layer(x).clone())
                assert impl.last_algo() == ran
            assert torch.equal(outs[-1], outs[-2]) or norm      # the tile does not change a product's sums
            torch.testing.assert_close(outs[-1], outs[-2], rtol=2 ** -9, atol=1e-6)
    bm, bn, _ = cfg.ALGO_TILES[algo]
    tiles = (M // bm) * (N // bn)
    for extra, ran in (({"search": "exhaustive", "raster_group": 2}, algo), ({}, chosen)):
        config = {"BM": bm, "BN": bn, "Algo": algo, "hint": list(range(tiles)), "cSeg": [tiles], **extra}
        layer = OverlapRowParallelLayer(0, 1, K, N, M, config, "all_reduce", [0] * 16)
        layer(x)
        assert layer.overlap_class.last_algo() == ran
    torch.cuda.synchronize()
    impl.check_status()


def test_measured_row_time_is_sane():
    from flashoverlap_b200.tune.runtime import gather_algo_candidates, measure_row_us, pick_algo_by_timing

    impl = make_overlap_impl(timeout_ms=3000)
    row_ar = measure_row_us(impl, 2048, "all_reduce", torch.float16, reps=3)
    row_rs = measure_row_us(impl, 2048, "reduce_scatter", torch.bfloat16, reps=3)
    assert 0.05 < row_ar < 200.0 and 0.05 < row_rs < 200.0   # microseconds per row and row group
    impl.check_status()
    # the timed tile pick returns one of its candidates and a time for each
    A = torch.randn(1024, 256, device="cuda", dtype=torch.float16)
    B = torch.randn(2048, 256, device="cuda", dtype=torch.float16)
    C = torch.empty(1024, 2048, device="cuda", dtype=torch.float16)
    cands = gather_algo_candidates(1024, 2048)[:3]
    best, timed = pick_algo_by_timing(lambda a: impl.allgather_gemm(A, B, C, a), cands, warmup=1, reps=2)
    assert best in cands and [a for a, _ in timed] == cands and all(t > 0 for _, t in timed)
    impl.check_status()
