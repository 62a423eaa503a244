"""Rules of the prompt path that the host decides, without a device."""
import ctypes as C
import os
import subprocess
import sys

import pytest

from k2t_internal import internal


def batches(n_tok, max_batch, experts):
    prompt_batch = internal("prompt_batch", C.c_uint32, C.c_size_t, C.c_size_t, C.c_uint32, C.c_bool)
    out, done = [], 0
    while done < n_tok:
        out.append(prompt_batch(n_tok, done, max_batch, experts))
        assert 0 < out[-1] <= min(n_tok - done, max_batch)
        done += out[-1]
    return out


@pytest.mark.parametrize("n,dense,experts", [
    (2, [2], None), (300, [300], None), (512, [512], None), (513, [512, 1], None), (544, [512, 32], None), (545, [512, 33], [384, 161]), (576, [512, 64], [384, 192]),
    (577, [384, 193], None), (1000, [512, 488], None), (1025, [512, 512, 1], None), (1100, [384, 384, 332], None), (1537, [512, 512, 512, 1], None),
    (1600, [512, 512, 512, 64], [512, 384, 384, 320]), (1700, [512, 512, 512, 164], [512, 512, 384, 292])])
def test_batches_of_a_prompt(n, dense, experts):
    assert batches(n, 512, False) == dense
    assert batches(n, 512, True) == (experts or dense)


@pytest.mark.parametrize("experts", [False, True])
@pytest.mark.parametrize("max_batch", [16, 48, 128, 208, 256, 384, 512])
def test_as_few_batches_as_there_can_be(max_batch, experts):
    for n in list(range(1, 3 * max_batch + 40)) + [4001, 8192, 20011]:
        b = batches(n, max_batch, experts)
        assert sum(b) == n and len(b) == -(-n // max_batch)
        assert all(x % 16 == 0 for x in b[:-1])


def in_process(code, **env):
    """stdout of a Python program with environment variables that the library reads once."""
    return subprocess.run([sys.executable, "-c", code], check=True, capture_output=True, text=True, cwd=os.path.dirname(os.path.abspath(__file__)),
                          env=dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path), **env)).stdout.strip()


@pytest.mark.parametrize("switch,want", [(None, "0 1 1"), ("0", "0 0 0"), ("200", "0 0 1")])
def test_expert_tiles_obey_the_tensor_core_switch(switch, want):
    """512 pairs of 8 experts as 8, 100 and 300 tokens: the grouped form is a tensor-core form."""
    code = ("import ctypes as C; from k2t_internal import internal; f = internal('experts_grouped', C.c_bool, *[C.c_uint32] * 6); "
            "print(*[int(f(t, 512, 8, 2048, 4096, 4)) for t in (8, 100, 300)])")
    assert in_process(code, **({} if switch is None else dict(KRONOS_CUDA_TC_MIN_TOKENS=switch))) == want


def test_largest_batch_of_the_prompt_gemm():
    """The padded tokens of the operand image are 32 to a CTA along grid.y, which ends at 65535: 2 097 025 tokens pad to 65536 x 32."""
    takes = internal("gemm_f16_takes", C.c_bool, C.c_size_t)
    assert [takes(n) for n in (0, 1, 16, 512, 2097024, 2097025, 2097120, 2097121, 2 ** 32 + 16)] == [False, True, True, True, True, False, False, False, False]
    for n in range(2096900, 2097200):
        assert takes(n) == ((n + 127) // 128 * 4 <= 65535)


# (rows, cols, tokens): the conversion launch pays / is not taken, with 148 SMs (of the last row, with rows of 128 chunks and more or 49152 of them, it would pay by now)
CONVERTED = [(6144, 2048, 33), (16384, 2048, 17), (49152, 2048, 17), (49152, 2048, 512), (2048, 2048, 200), (3584, 18944, 65), (4608, 3584, 100), (1536, 576, 512)]
DIRECT = [(64, 192, 16), (960, 576, 100), (1536, 576, 200), (960, 576, 512), (1024, 192, 512), (2048, 2048, 128), (6144, 2048, 32), (16384, 2048, 16), (4608, 3584, 64),
          (2048, 8192, 128), (49152, 2048, 16), (3584, 18944, 64)]


def test_which_batches_are_converted():
    pays = internal("gemm_f16_pays", C.c_bool, C.c_uint32, C.c_uint32, C.c_size_t, C.c_int)
    assert [x for x in CONVERTED if not pays(x[0], x[1] // 64, x[2], 148)] == []
    assert [x for x in DIRECT if pays(x[0], x[1] // 64, x[2], 148)] == []
    assert all(pays(rows, nc, n, 148) for rows in (64, 49152) for nc in (1, 300) for n in (16 * 0xFFFF + 1, 2000000))          # more than the integer GEMM takes


# experts, routes, width, bits: tokens at which a GEMV per pair was faster, at which tiles were (2048 columns)
@pytest.mark.parametrize("n_experts,k,d_ff,bits,gemv,tiles", [
    (128, 8, 768, 3, (16, 24, 32), (48, 56, 64, 72, 128)), (128, 8, 768, 4, (16, 20), (28, 32, 48, 64)), (128, 8, 768, 5, (), (16, 20, 32, 64)), (128, 8, 768, 2, (), (16, 32, 64)),
    (64, 6, 768, 3, (16, 20, 24), (32, 40, 56, 64)), (64, 6, 768, 4, (16,), (24, 32, 48)), (64, 6, 768, 5, (), (16, 24)), (64, 6, 768, 2, (), (16, 24)),
    (64, 6, 1408, 3, (16, 24, 32), (40, 48, 64, 80)), (16, 4, 2816, 3, (), (16, 20, 24, 32)), (16, 4, 2816, 4, (), (16, 20)), (16, 4, 2816, 5, (), (16,)),
    (8, 2, 4096, 4, (), (16, 20, 32)), (4, 2, 2048, 3, (), (16, 20, 32, 48)), (256, 8, 768, 2, (), (16, 32))])
def test_experts_take_the_faster_form(n_experts, k, d_ff, bits, gemv, tiles):
    grouped = internal("experts_grouped", C.c_bool, *[C.c_uint32] * 6)
    form = {t: grouped(t, t * k, n_experts, 2048, d_ff, bits) for t in gemv + tiles}
    assert form == {**dict.fromkeys(gemv, False), **dict.fromkeys(tiles, True)}


# heads, kv heads, head size, tokens, context: where the row-sharing attention was slower, where it was faster
SLOWER = [(32, 32, 64, 16, 384), (32, 32, 64, 32, 1024), (32, 32, 64, 16, 6400), (9, 3, 64, 16, 512), (9, 3, 64, 48, 640), (9, 3, 64, 64, 3072), (9, 3, 64, 64, 6400),
          (28, 4, 128, 16, 1536), (28, 4, 128, 16, 6400)]
FASTER = [(32, 32, 64, 16, 128), (32, 32, 64, 32, 384), (32, 32, 64, 48, 640), (32, 32, 64, 64, 6400), (32, 32, 64, 512, 6400), (9, 3, 64, 16, 384), (9, 3, 64, 64, 640),
          (9, 3, 64, 128, 2432), (9, 3, 64, 256, 6400), (28, 4, 128, 16, 768), (28, 4, 128, 32, 1152), (28, 4, 128, 64, 6400), (28, 4, 128, 512, 6400), (32, 4, 128, 32, 3584)]


def test_which_batches_share_rows():
    pays = internal("attention_prompt_pays", C.c_bool, *[C.c_uint32] * 5)
    ask = lambda q, kv, d, n, ctx: pays(n, q, kv, d, ctx)  # noqa: E731
    assert [x for x in SLOWER if ask(*x)] == [] and [x for x in FASTER if not ask(*x)] == []
    assert not any(ask(32, 4, 128, n, 128) for n in range(1, 16))


def test_rows_of_an_attention_tile():
    """Scores of 16 rows take 64 bytes per position (rounded up to 16), beside the queries and outputs, in 220 KB."""
    rows = internal("attention_prompt_rows", C.c_uint32, C.c_uint32, C.c_uint32)
    last = lambda d, r: max(ctx for ctx in range(128, 8192) if rows(d, ctx) >= r)  # noqa: E731
    assert [last(64, 16), last(128, 16), last(64, 8), last(128, 8)] == [3424, 3344, 6944, 6864]
    assert rows(96, 128) == 0


class RouterArgs(C.Structure):
    _fields_ = [("w", C.c_void_p), ("bias", C.c_void_p), ("x", C.c_void_p), ("n_experts", C.c_uint32), ("hidden", C.c_uint32), ("top_k", C.c_uint32), ("norm_topk", C.c_int32),
                ("scoring", C.c_uint32), ("route_ids", C.c_void_p), ("route_w", C.c_void_p), ("logits", C.c_void_p), ("done", C.c_void_p), ("route_stride", C.c_uint32),
                ("staged", C.c_uint32), ("err_flag", C.c_void_p)]


# hidden, experts: tokens at which one launch was faster, at which two were
@pytest.mark.parametrize("hidden,n_experts,one,two", [
    (512, 64, (16, 64, 200), (256, 512)), (1024, 8, (16, 512), ()), (1024, 64, (16, 128, 200), (256, 300)), (1024, 128, (16, 64, 96), (128, 512)), (1536, 64, (16, 200), (256, 400)),
    (1536, 256, (16, 48), (64, 128)), (2048, 16, (16, 512), ()), (2048, 32, (16, 300), (512,)), (2048, 64, (16, 128, 200), (300, 512)), (2048, 128, (16, 24, 48, 64, 96), (128, 300, 512)),
    (2048, 256, (16, 48), (64, 128)), (2560, 64, (16, 160), (200, 300)), (3072, 64, (16, 160), (256, 300)), (3072, 128, (16, 96), (128, 200)), (3584, 128, (16, 64), (96, 128)),
    (4096, 64, (16, 96, 128), (200, 300)), (4096, 128, (16, 64), (96, 200)), (5120, 128, (16, 64), (96, 128)), (6144, 64, (16, 256), (300, 512)), (7168, 128, (16, 128), (160, 300)),
    (8192, 256, (16, 64), (96, 128))])
def test_router_takes_the_faster_form(hidden, n_experts, one, two):
    in_two = internal("router_in_two", C.c_bool, C.POINTER(RouterArgs), C.c_uint32)
    a = RouterArgs(w=256, x=256, n_experts=n_experts, hidden=hidden, top_k=min(8, n_experts))
    assert {t: in_two(C.byref(a), t) for t in one + two} == {**dict.fromkeys(one, False), **dict.fromkeys(two, True)}
    assert not any(in_two(C.byref(a), t) for t in range(1, 16))


# format, rows, columns: tokens at which the GEMM of shorter rows was faster, at which the one of long rows was (148 SMs; rows of a whole pass of 32 chunks and a part)
FMT = dict(b4=0, b5=1, b6=2, nf4=3, nf3=4, nf5=5)


@pytest.mark.parametrize("fmt,rows,cols,short,long", [
    ("b5", 4608, 3584, (16, 77, 256), (300, 512)), ("b5", 3584, 3584, (16, 300), (400, 512)), ("b5", 2880, 2880, (16, 300), (400,)), ("b5", 4096, 4096, (), (16, 512)), ("b5", 3584, 18944, (), (16, 77, 512)),
    ("b5", 12288, 3584, (32, 64), (96, 512)), ("nf5", 3584, 3584, (16, 160), (200, 512)), ("nf5", 4096, 7168, (32, 128), (160, 512)), ("nf5", 3584, 18944, (32, 160), (200, 512)), ("nf5", 2048, 8192, (), (16, 512)), ("nf3", 3584, 3584, (32, 160), (200, 512)),
    ("nf3", 4096, 7168, (), (16, 512)), ("nf4", 4096, 2880, (32, 128), (160, 512)), ("nf4", 2048, 3584, (32, 256), (300, 512)), ("nf4", 2048, 4096, (), (16, 300)), ("b6", 4608, 3584, (), (16, 512)),
    ("b4", 37888, 3584, (), (16, 77)), ("b5", 260, 4160, (16, 512), ()), ("nf4", 960, 1984, (16, 512), ())])
def test_long_rows_take_the_faster_kernel(fmt, rows, cols, short, long):
    takes = internal("gemm_prompt_takes", C.c_bool, C.c_int, C.c_uint32, C.c_uint32, C.c_uint32, C.c_int)
    assert {t: takes(FMT[fmt], rows, cols // 64, t, 148) for t in short + long} == {**dict.fromkeys(short, False), **dict.fromkeys(long, True)}
