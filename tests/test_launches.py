"""Which kernels a call launches, with which grid and in which order, by the library linked with a runtime that runs nothing."""
import ctypes as C
import re

import numpy as np
import pytest

from host_runtime import Library, build
from test_gpu_quant import Q8_SHAPES, SPLIT_SIZES
from zignn_b200 import ggml, hostmodel, structs

ACT_F32, ACT_Q8, ERR_CUDA, ERR_LIMIT = 0, 1, 3, 5


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return Library(build(tmp_path_factory.mktemp("launches")))


def u32(values):
    return np.ascontiguousarray(values, np.uint32)


def pointer(a):
    return a.ctypes.data_as(C.c_void_p)


LENISUN = dict(architecture="Lenisun", vocab=64, width=64, norm=dict(eps=1e-6), embedding=dict(scale=1.0), layers=[
    dict(type="attention", mixer=dict(heads=2, kv_heads=1, dim=32, vdim=32, scale=0.2), mlp=dict(kind="dense", ff=64, limit=2.0))] * 2)


def decoder(library, ctx=64, n_seq=3):
    host = hostmodel.LenisunHost.synthetic(LENISUN, seed=1, std=0.2)
    cfg, weights, engine = host.config_struct(ctx, n_seq, False), host.weights_struct(), C.c_void_p()
    assert library.lib.zq_decoder_create(C.byref(cfg), C.byref(weights), None, C.byref(engine)) == 0
    return engine


def test_a_step_starts_when_its_rows_are_set(library):
    """Kernels of a step read its positions and slots ahead of their wait, so its first kernel is no dependent launch; the others
    are."""
    engine, lg, lib = decoder(library), C.c_void_p(), library.lib
    calls = [lambda: lib.zq_decoder_decode_next(engine, 0, 5, None, C.byref(lg)),
             lambda: lib.zq_decoder_decode_next_batch(engine, pointer(u32([2, 0])), pointer(u32([1, 2])), 2, None, C.byref(lg)),
             lambda: lib.zq_decoder_decode_next_batch(engine, pointer(u32([2, 0, 1])), pointer(u32([1, 2, 3])), 3, None, C.byref(lg)),
             lambda: lib.zq_decoder_decode_greedy(engine, 1, 5, 1, None, pointer(u32([0]))),
             lambda: lib.zq_decoder_extend(engine, 1, pointer(u32([7])), 1, None, 0, None, None)]
    for call in calls:
        seen, status = library.launches(call)
        assert status == 0 and any("gqa_decode" in l.name for l in seen)
        assert "set_row" in seen[0].name or "set_step_rows" in seen[0].name
        assert not seen[0].dependent and not seen[1].dependent, [l.name for l in seen]
        assert all(l.dependent for l in seen[2:] if "feed_row" not in l.name and "argmax" not in l.name), [(l.name, l.dependent) for l in seen]
    lib.zq_decoder_free(engine)


def weight(library, qtype, n, k):
    raw, w = np.zeros(ggml.tensor_bytes(qtype, n * k), np.uint8), C.c_void_p()
    assert library.lib.zq_weight_upload(pointer(raw), qtype, n, k, None, C.byref(w)) == 0
    return w


def matmul(library, w, m, act):
    """Launches and status of a product; nothing reads its operands."""
    lib, somewhere = library.lib, C.c_void_p(1 << 20)
    size = lib.zq_matmul_workspace_bytes(w, m, act)
    return library.launches(lambda: lib.zq_matmul(w, somewhere, somewhere, m, act, None, somewhere, size, None))


@pytest.mark.parametrize("n", [8, 64, 128, 160, 300])
def test_q8_rows_up_to_the_limit_of_a_grid(library, n):
    """65535 CTAs of 64 rows, whatever the count of weight rows; what goes beyond is refused."""
    w = weight(library, ggml.Q8_0, n, 32)
    for m in (2097120, 2097121, 4194240):
        seen, status = matmul(library, w, m, ACT_Q8)
        assert status == 0 and "gemm_q8_kernel" in seen[-1].name and seen[-1].grid[1] <= 65535, (m, status)
    assert matmul(library, w, 4194241, ACT_Q8)[1] == ERR_LIMIT
    library.lib.zq_weight_free(w)


@pytest.mark.parametrize("qtype", [ggml.Q4_0, ggml.Q4_1, ggml.Q8_0])
def test_sizes_of_the_q8_product_test_take_every_shape(library, qtype):
    """Of test_gpu_quant.py: (warps, weight tiles per warp, column tiles) of the kernel that each of its sizes launches on 148 SMs."""
    taken = set()
    for n, k, m in Q8_SHAPES[qtype]:
        w = weight(library, qtype, n, k)
        name = matmul(library, w, m, ACT_Q8)[0][-1].name
        taken.add(tuple(int(v) for v in re.search(r"gemm_q8_kernelILi\d+ELi(\d+)ELi(\d+)ELi(\d+)E", name).groups()))
        library.lib.zq_weight_free(w)
    assert taken == {(8, 1, 8), (4, 2, 4), (4, 1, 4), (4, 1, 2), (4, 1, 1)}


def split_tile(library, qtype, n, k, m):
    """(weight rows, activation rows, quads of K per step, stages) of the f32-accurate product that the call launches."""
    w = weight(library, qtype, n, k)
    name = matmul(library, w, m, ACT_F32)[0][-1].name
    library.lib.zq_weight_free(w)
    wr, ks, nt, d = (int(v) for v in re.search(r"gemm_split_kernelILi\d+ELi(\d+)ELi(\d+)ELi(\d+)ELi(\d+)E", name).groups())
    return wr * 16, nt * 8, ks, d


@pytest.mark.parametrize("qtype", [ggml.Q4_0, ggml.Q4_1, ggml.Q8_0])
def test_sizes_of_the_split_product_test_take_every_tile(library, qtype):
    assert {split_tile(library, qtype, n, k, m) for n, k, m in SPLIT_SIZES} == {
        (16, 16, 8, 2), (32, 16, 4, 3), (32, 24, 4, 3), (32, 32, 4, 2), (64, 24, 2, 4), (64, 32, 2, 4), (64, 48, 2, 3), (128, 48, 1, 2),
        (64, 24, 2, 2), (64, 32, 2, 2)}


@pytest.mark.parametrize("n", [9473, 11000, 12160])
def test_split_product_of_more_tiles_than_sms_takes_two_per_sm(library, n):
    """21 to 32 rows: two CTAs per SM of a tile that holds the rows once, not one CTA of 48 columns (14.4 and 17.1 us against 23.0)."""
    for m in (21, 24, 25, 32):
        assert split_tile(library, ggml.Q4_0, n, 1152, m) == (64, 24 if m <= 24 else 32, 2, 2), m
    assert split_tile(library, ggml.Q4_0, 4096, 6144, 32) == (32, 32, 4, 2)


@pytest.mark.parametrize("heads,kv_heads,dim,ctx,slots,ranges", [
    (12, 4, 64, 2048, 1, 32), (12, 4, 64, 2048, 6, 16), (12, 4, 64, 2048, 16, 8), (12, 4, 64, 2048, 64, 8), (12, 4, 64, 256, 1, 1),
    (8, 2, 128, 2048, 6, 32), (8, 2, 128, 2048, 8, 16), (8, 2, 128, 2048, 64, 8), (8, 2, 128, 256, 8, 4), (8, 2, 128, 256, 16, 1),
    (4, 1, 256, 2048, 1, 32), (4, 1, 256, 2048, 64, 32), (4, 1, 256, 256, 64, 4), (12, 4, 64, 8192, 64, 32), (12, 4, 64, 1500, 1, 24)])
def test_ranges_of_the_decode_attention(library, heads, kv_heads, dim, ctx, slots, ranges):
    """By the cache alone: any count of rows of a step cuts a row's keys alike. No second kernel behind one range."""
    g, somewhere, lib = structs.Gqa(heads, kv_heads, dim, dim, ctx, slots, 1.0, 1e-6, 0.0, 0.0), C.c_void_p(1 << 20), library.lib
    for rows in (1, 2, slots):
        seen, status = library.launches(lambda: lib.zq_gqa_attention(C.byref(g), *[somewhere] * 6, rows, 0, 0, somewhere, 0, None))
        assert status == 0 and "gqa_decode" in seen[0].name and seen[0].grid == (ranges, kv_heads, rows)
        assert len(seen) == (1 if ranges == 1 else 2)


@pytest.mark.parametrize("rows,heads,alone", [(1, 4, True), (37, 4, True), (38, 4, False)])
def test_plain_attention_has_an_sm_per_cta(library, rows, heads, alone):
    """f32: as long as the CTAs are no more than the SMs, no two of them fit one."""
    g, somewhere, lib = structs.Gqa(heads, 1, 64, 64, 256, rows, 1.0, 1e-6, 0.0, 0.0), C.c_void_p(1 << 20), library.lib
    seen, status = library.launches(lambda: lib.zq_gqa_attention(C.byref(g), *[somewhere] * 6, rows, 0, 0, somewhere, 1, None))
    assert status == 0 and "gqa_plain" in seen[0].name
    assert (2 * (seen[0].smem + 1024) > 228 * 1024) == alone, seen[0].smem


@pytest.mark.parametrize("n,k,m", [(1152, 6912, 2), (1152, 6912, 16), (1152, 6912, 17), (768, 768, 16), (1184, 1024, 8), (64, 64, 9)])
def test_few_ctas_of_the_q8_product_have_an_sm_each(library, n, k, m):
    """With K over the warps or not: no two CTAs of a grid of at most 148 fit one SM."""
    w = weight(library, ggml.Q8_0, n, k)
    product = matmul(library, w, m, ACT_Q8)[0][-1]
    library.lib.zq_weight_free(w)
    assert product.grid[0] * product.grid[1] <= 148 and 2 * (product.smem + 1024) > 228 * 1024, (product.name, product.grid, product.smem)


def test_a_step_of_several_sequences_is_refused_while_its_stream_captures(library):
    """It advances the host's lengths, so a recording could not be replayed: nothing is launched and no length changes."""
    engine, lg, lib, n = decoder(library), C.c_void_p(), library.lib, C.c_uint32()
    step = lambda: lib.zq_decoder_decode_next_batch(engine, pointer(u32([2, 0])), pointer(u32([1, 2])), 2, None, C.byref(lg))
    lib.set_capturing(1)
    seen, status = library.launches(step)
    lib.set_capturing(0)
    assert status == ERR_CUDA and not seen
    assert lib.zq_decoder_seq_len_of(engine, 2, C.byref(n)) == 0 and n.value == 0
    assert step() == 0 and lib.zq_decoder_seq_len_of(engine, 2, C.byref(n)) == 0 and n.value == 1
    lib.zq_decoder_free(engine)


@pytest.mark.parametrize("rows,kernels", [(256, 1), (257, 2), (300, 2), (600, 3)])
def test_rows_of_a_step_in_portions(library, rows, kernels):
    engine, lg, lib = decoder(library, n_seq=rows), C.c_void_p(), library.lib
    seen, status = library.launches(lambda: lib.zq_decoder_decode_next_batch(
        engine, pointer(u32(range(rows))), pointer(u32([1] * rows)), rows, None, C.byref(lg)))
    assert status == 0 and ["set_step_rows" in l.name for l in seen[:kernels + 1]] == [True] * kernels + [False]
    assert not seen[kernels].dependent
    lib.zq_decoder_free(engine)
