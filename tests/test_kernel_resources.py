"""Resource usage of the hot kernels as ptxas reports it at build time (no GPU needed).

A by-reference lambda that stops being inlined, or a locally indexed array, moves a kernel's working set into a stack
frame; the GEMM then loses a third of its speed without any functional symptom. The build keeps ptxas' report, this
test reads it."""
import pytest

from openvino_b200 import build


@pytest.fixture(scope="module")
def gemm():
    build.build_cuda()
    res = build.kernel_resources("gemm_sm100")
    if not res:
        build.build_cuda(force=True)
        res = build.kernel_resources("gemm_sm100")
    assert res, "no ptxas report for gemm_sm100.cu"
    return res


def test_gemm_variants_have_no_stack_working_set(gemm):
    assert len(gemm) >= 25                     # 5 token-tile sizes x 5 weight formats
    for name, r in gemm.items():
        assert r["stack"] <= 64, (name, r)     # a few words for the bounded-wait helper are fine; hundreds of bytes are not
        assert r["spill_stores"] <= 16 and r["spill_loads"] <= 32, (name, r)


def test_decode_variants_fit_two_ctas_per_sm(gemm):
    # decode-sized quantised tiles run two CTAs of 352 threads per SM: at most 65536 / 704 = 93 registers per thread
    small = [r for n, r in gemm.items() if r["registers"] <= 93]
    assert len(small) >= 9                     # u4 / u8 / fp8 at 16, 32 and 64 tokens


def test_gemm_uses_no_static_shared_memory(gemm):
    # the kernel opts in to the whole dynamic shared-memory limit of the SM: one static __shared__ word makes the opt-in fail
    assert all(r["static_smem"] == 0 for r in gemm.values()), {n: r["static_smem"] for n, r in gemm.items() if r["static_smem"]}


def test_layered_decoders_need_no_more_than_the_full_library(gemm):
    assert all((build.CSRC / "cuda" / (stem + ".cu")).exists() for stem in build.LAYERED_STEMS)
    assert build.layered_library() == build.LIB / "libovb_cuda.so"        # built and current: nothing else is compiled


@pytest.mark.parametrize("stem", ["attention_latent", "attention_sm100", "residual", "attention_heads", "gemm_f32", "attention_exact", "delta_rule"])
def test_kernels_of_layered_decoders_do_not_spill(gemm, stem):
    res = build.kernel_resources(stem)
    # kernels that are held to a register limit for the sake of occupancy may park a few words outside their loops
    words = 16 if stem in ("attention_heads", "delta_rule") else 0
    assert res and all(r["spill_stores"] <= 4 * words and r["stack"] <= 4 * words for r in res.values()), \
        {n: r for n, r in res.items() if r["spill_stores"] or r["stack"]}


@pytest.mark.parametrize("T,B,Hq,Hkv,two", [
    (48 + 16, 49, 32, 8, 0), (40 + 64, 41, 32, 8, 0), (40 + 512, 41, 32, 8, 0), (64 * 20, 64, 32, 8, 0), (30 + 300, 31, 64, 8, 0),     # mostly decoding, short
    (40 + 2048, 41, 32, 8, 1), (8191, 1, 32, 8, 1), (8 * 1024, 8, 32, 8, 1), (40 * 33, 40, 32, 8, 1), (2048, 1, 64, 8, 1),             # full tiles
    (1, 1, 32, 8, 0), (1000, 1, 32, 8, 0), (3 * 333, 3, 32, 8, 0),                                                                    # too few tiles
])
def test_two_query_tiles_go_to_steps_of_full_tiles(gemm, T, B, Hq, Hkv, two):
    from openvino_b200.ops import cuda as ops
    assert ops.lib().ovb_pa_two_query_tiles(T, B, Hq, Hkv) == two


@pytest.mark.parametrize("fmt,N,K,T,expanded", [
    ("u4", 4096, 14336, 1024, 0), ("u4", 57344, 8192, 1024, 0), ("u4", 8192, 28672, 1024, 0), ("u4", 8192, 28672, 8192, 0), ("u8", 8192, 28672, 1024, 0),
    ("f8", 8192, 28672, 1024, 0), ("u4", 10240, 8192, 1280, 0),
    ("u4", 28672, 4096, 1024, 1), ("u4", 28672, 4096, 8192, 1), ("u4", 57344, 8192, 4096, 1), ("u8", 4096, 14336, 1024, 1), ("f8", 8192, 28672, 2048, 1),
    ("u8", 28672, 4096, 1024, 1), ("u8", 28672, 4096, 1023, 0)])
def test_weights_are_expanded_where_that_is_faster(gemm, fmt, N, K, T, expanded):
    """Both sides of the rule at sizes that were measured on both kernels."""
    import ctypes as C
    from openvino_b200.ops import cuda as ops
    a = ops.GemmArgs()
    a.T, a.N, a.K, a.ldx, a.group_size, a.wmode = T, N, K, K, 128, {"u4": ops.W_U4, "u8": ops.W_U8, "f8": ops.W_F8}[fmt]
    a.act = ops.ACT_SWIGLU if N in (28672, 57344) else ops.ACT_NONE
    a.x = a.w = a.out = 16
    assert (ops.lib().ovb_gemm_scratch_bytes(C.byref(a)) > 0) == bool(expanded)


@pytest.mark.parametrize("N,K,T,route", [(8192, 28672, 4, 0), (57344, 28672, 4, 0), (8192, 28672, 3, 2), (1024, 28672, 4, 2), (4096, 14336, 4, 2), (128256, 4096, 1, 2),
                                         (4096, 4096, 5, 0)])
def test_few_tokens_leave_clusters_that_would_share_many_tiles(gemm, N, K, T, route):
    import ctypes as C
    from openvino_b200.ops import cuda as ops
    a = ops.GemmArgs()
    a.x = a.w = a.out = 16
    a.T, a.N, a.K, a.ldx, a.group_size, a.wmode = T, N, K, K, 128, ops.W_U4
    assert ops.lib().ovb_gemm_route(C.byref(a)) == route


def test_step_descriptors_have_the_size_of_the_c_structs(gemm):
    import ctypes as C
    import struct
    from openvino_b200.ops import cuda as ops
    sizes = [struct.calcsize("<" + ops.LLM_WEIGHT), struct.calcsize(ops.LLM_LAYER), C.sizeof(ops.LlmStep)]
    assert [ops.lib().ovb_llm_struct_bytes(i) for i in range(3)] == sizes
    assert C.sizeof(dict(ops.LlmStep._fields_)["head"]) == sizes[0]


SINGLE, PAIR, STREAM, RING, FEW = range(5)


@pytest.mark.parametrize("fmt,N,K,splits,T,kernel", [
    # what the test of the few-token kernel runs with a number of splits: one stage of K, odd shares of K, several rounds of tiles
    *[(f, N, K, s, T, FEW) for f, T in (("u4", 5), ("u8", 33), ("f8", 64))
      for N, K, splits in ((128, 256, (1,)), (256, 1280, (2, 3, 5)), (512, 2048, (4, 6, 7, 8)), (128 * 150, 256, (1,)), (128 * 76, 512, (2,)), (128 * 19, 2048, (8,))) for s in splits],
    # both sides of the rule, at sizes that were measured on both kernels
    ("u4", 128256, 4096, 0, 16, FEW), ("u4", 4096, 14336, 0, 16, FEW), ("u4", 28672, 1024, 0, 16, SINGLE), ("u4", 4096, 1024, 0, 16, FEW), ("u4", 4096, 2048, 0, 37, SINGLE),
    ("u4", 28672, 4096, 0, 37, FEW), ("u4", 4096, 4096, 0, 37, FEW), ("u4", 20480, 1024, 0, 37, SINGLE), ("u4", 128256, 4096, 0, 64, SINGLE),
    ("u8", 6144, 4096, 0, 24, FEW), ("u8", 1024, 1024, 0, 24, SINGLE), ("u8", 24576, 2048, 0, 48, SINGLE), ("f8", 8192, 28672, 0, 64, FEW), ("f8", 1024, 1024, 0, 64, SINGLE),
    ("u8", 28672, 4096, 0, 64, SINGLE), ("u8", 128256, 4096, 0, 64, FEW), ("f8", 10240, 8192, 0, 37, SINGLE), ("f8", 10240, 14336, 0, 37, FEW),
    ("u4", 512, 2048, 0, 65, SINGLE), ("u4", 512, 2048 + 128, 0, 16, SINGLE), ("u4", 512 + 32, 2048, 0, 16, SINGLE),
    ("u4", 2048, 4096, 0, 1, RING), ("u4", 2048, 4096, 0, 4, RING), ("u4", 2048, 4096, 0, 5, FEW), ("u4", 2048, 4096 - 256, 0, 1, STREAM), ("u4", 1280, 8192, 0, 3, RING),
    ("u8", 512, 2048, 0, 4, STREAM), ("f8", 512, 2048, 0, 4, STREAM), ("u8", 128256, 4096, 0, 4, FEW), ("dense", 512, 2048, 0, 8, STREAM), ("dense", 512, 2048, 0, 9, SINGLE),
    ("dense", 28672, 4096, 0, 512, PAIR)])
def test_products_run_on_the_kernel_for_their_size(gemm, fmt, N, K, splits, T, kernel):
    """Which kernel the products run on that the kernels' own tests compute."""
    import ctypes as C
    from openvino_b200.ops import cuda as ops
    a = ops.GemmArgs()
    a.x = a.w = a.out = a.scales = 16
    a.T, a.N, a.K, a.ldx, a.group_size, a.splits = T, N, K, K, 128, splits
    a.wmode = {"u4": ops.W_U4, "u8": ops.W_U8, "f8": ops.W_F8, "dense": ops.W_BF16}[fmt]
    a.w_tiled = 1 if fmt == "dense" else 0
    assert ops.lib().ovb_gemm_kernel(C.byref(a)) == kernel
