"""Which kernel a call goes to, where the sizes decide it on the host: no GPU is needed."""
import pytest

from vitna_anchor_b200 import ops


# (tokens, q and k heads, v heads, their sizes, taps): what the slices of channels were measured to be slower or faster at than a block a token
@pytest.mark.parametrize("sizes,sliced", [
    ((64, 16, 32, 128, 128, 4), False), ((65, 1, 2, 16, 16, 4), False), ((400, 2, 4, 32, 64, 4), False), ((592, 2, 2, 20, 12, 4), False), ((1183, 2, 2, 20, 12, 4), False),
    ((200, 3, 9, 64, 64, 4), False), ((65, 3, 9, 64, 64, 2), False), ((400, 1, 1, 512, 64, 4), False), ((400, 1, 1, 1024, 64, 4), False), ((4000, 1, 2, 64, 64, 5), False),
    ((65, 4, 16, 128, 128, 4), True), ((400, 3, 9, 64, 64, 4), True), ((600, 2, 4, 32, 64, 4), True), ((600, 1, 1, 1024, 64, 4), True), ((1185, 1, 2, 16, 16, 4), True)])
def test_delta_rule_preparation(sizes, sliced):
    assert (ops.lib().vk_delta_prepare_slices(*sizes) > 0) == sliced


# (rows, columns, K), into a sum or not: where the few-rows tcgen05 product was measured to be slower, or less exact, than what stands in, and where it is the faster one
@pytest.mark.parametrize("sizes,acc,taken", [
    ((8, 16384, 1536), False, False), ((4, 12800, 1920), False, False), ((8, 6144, 2048), False, False), ((16, 2048, 2048), False, False), ((16, 4096, 1024), False, False),
    ((12, 5120, 960), False, False), ((32, 2112, 1024), False, False), ((28, 2048, 2048), True, False), ((40, 16384, 1536), False, False), ((64, 1024, 1056), False, False), ((33, 1536, 1536), False, False), ((32, 1600, 960), False, False), ((64, 768, 2048), True, False),
    ((64, 49152, 576), False, False), ((40, 49152, 960), False, False), ((64, 131072, 192), False, False), ((8, 131072, 192), False, False), ((64, 16384, 2048), True, False),
    ((64, 2048, 1000), False, False), ((64, 6144, 2056), False, False), ((64, 576, 576), False, False),
    ((1, 49152, 576), False, True), ((8, 49152, 960), False, True), ((16, 49152, 2048), False, True), ((16, 2048, 8192), True, True), ((64, 6144, 2048), False, True),
    ((64, 2048, 8192), True, True), ((64, 2048, 2048), True, True), ((64, 16384, 2048), False, True), ((64, 1600, 960), False, True), ((32, 49152, 960), False, True), ((16, 5120, 960), False, True), ((17, 2560, 2560), True, True),
    ((17, 1536, 4096), True, True), ((33, 1600, 960), False, True), ((33, 960, 2560), True, True), ((32, 22016, 4096), False, True)])
def test_few_rows_products(sizes, acc, taken):
    assert ops.rows_tcgen05_sizes(*sizes, acc) == taken


# (kind, rows, columns, K) as vk_linear_tcgen05_route has them: where the wide tiles, or pairs of blocks, were measured to be slower, and where they are the faster ones
@pytest.mark.parametrize("sizes,route", [
    ((0, 8192, 790, 272), 0), ((0, 1301, 1746, 576), 0), ((0, 16384, 14678, 112), 0), ((2, 8192, 790, 272), 160), ((2, 16384, 1746, 576), 160), ((2, 16384, 6104, 256), 0),
    ((3, 8192, 1536, 576), 192), ((3, 16384, 3072, 768), 256), ((1, 16384, 1746, 576), 256), ((1, 1000, 4096, 4096), 256), ((2, 1301, 2560, 4096), 256), ((2, 4096, 674, 3536), 192),
    ((0, 8192, 6144, 2048), 257), ((3, 8192, 8192, 2048), 257), ((2, 8192, 2048, 8192), 257), ((2, 2048, 2048, 8192), 257), ((0, 3000, 1001, 1000), 192), ((0, 1301, 1352, 4656), 160), ((1, 1000, 1178, 4472), 160), ((0, 1301, 960, 2560), 0),
    ((4, 8192, 6144, 2048), 257), ((5, 8192, 2560, 2048), 257), ((1, 3000, 960, 4096), 161)])
def test_wide_products(sizes, route):
    assert ops.lib().vk_linear_tcgen05_route(*sizes) == route


# (rows, columns, type of the result: 0 float32, 1 bfloat16): where a warp a row was measured to be slower than eight rows a block, and where it is the faster one
@pytest.mark.parametrize("sizes,warps", [
    ((3000, 64, 1), False), ((4096, 256, 0), False), ((3000, 576, 1), False), ((3552, 640, 1), False), ((3200, 644, 1), False), ((7000, 640, 1), False), ((16384, 644, 1), False), ((16384, 768, 1), False),
    ((16384, 576, 0), False), ((16, 2052, 1), False),
    ((64, 2048, 1), True), ((1, 576, 1), True), ((2048, 576, 1), True), ((3000, 576, 0), True), ((4096, 576, 1), True), ((2048, 960, 1), True), ((8192, 2048, 1), True), ((16384, 960, 1), True)])
def test_norms(sizes, warps):
    assert bool(ops.lib().vk_rmsnorm_warp_blocks(*sizes)) == warps


# (tiles, heads, window, context): the groups of the prompt attention's form for heads of 64, and the parts that a walk may be cut into
@pytest.mark.parametrize("sizes,groups,parts", [
    ((16, 32, 0, 2048), 2, 1), ((64, 32, 0, 8192), 2, 1), ((41, 9, 0, 5200), 4, 1), ((42, 9, 0, 5300), 2, 1), ((16, 9, 0, 2048), 4, 1), ((1, 9, 0, 6100), 4, 6), ((8, 32, 0, 1024), 4, 1),
    ((32, 32, 0, 16), 1, 1), ((8, 20, 0, 128), 2, 1), ((32, 32, 64, 4096), 1, 1), ((3, 9, 64, 300), 2, 1), ((4, 20, 256, 3128), 2, 1), ((12, 9, 256, 1536), 2, 1), ((4, 20, 2000, 3128), 4, 3)])
def test_prompt_attention(sizes, groups, parts):
    assert ops.lib().vk_attention_prefill_plan(*sizes) == groups + 16 * parts
