"""CPU-side checks of the C-ABI library: it loads, exports every symbol the headers declare, the
host-only entry points compute the same indices as the oracle, and shape guards reject bad
shapes before any launch (no GPU needed: none of these calls touches a device)."""
import ctypes as C
import os
import re

import numpy as np
import pytest

import oracle_lib as O
from logismos_b200._lib import lib, library_path

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    names = set()
    for h in sorted(os.listdir(os.path.join(ROOT, "include"))):
        text = open(os.path.join(ROOT, "include", h)).read()
        text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
        names |= set(re.findall(r"\b((?:lg|logismos)_[a-z0-9_]+)\s*\(", text))
    return names


def test_library_exports_every_declared_symbol():
    assert os.path.exists(library_path()), "run python -m logismos_b200.build"
    dll = C.CDLL(library_path())
    syms = declared_symbols()
    assert len(syms) > 50
    missing = [s for s in sorted(syms) if not hasattr(dll, s)]
    assert not missing, missing


def test_the_four_reference_launcher_symbols_keep_their_names():
    dll = C.CDLL(library_path())
    for s in ("logismos_launch_matmul_naive_fp16", "logismos_launch_matmul_wmma_fp16", "logismos_launch_rms_norm_fp16",
              "logismos_launch_softmax_fp16", "logismos_launch_rope_fp16"):
        assert hasattr(dll, s)


def test_launcher_shape_guards_reject_without_launching():  # matmul/mod.rs:213-247, rope/mod.rs:215-269
    z = C.c_void_p(0)
    assert lib.logismos_launch_matmul_naive_fp16(z, z, z, 0, 4, 4, z) == 1
    assert lib.logismos_launch_matmul_naive_fp16(z, z, z, -1, 4, 4, z) == 1
    assert lib.logismos_launch_matmul_naive_fp16(z, z, z, 65536, 65536, 4, z) == 1   # M*N > i32::MAX
    assert lib.logismos_launch_matmul_wmma_fp16(z, z, z, 24, 16, 16, z) == 1         # not multiples of 16
    assert lib.logismos_launch_rope_fp16(z, z, 2**31 - 1, 2**31 - 1, 2, 2, z) == 1    # product overflows i64
    assert lib.logismos_launch_rope_fp16(z, z, 46341, 46341, 1, 2, z) == 1            # > i32::MAX
    assert lib.logismos_launch_rope_fp16(z, z, 1, 1, 1, 0, z) == 1
    assert lib.logismos_launch_rms_norm_fp16(z, z, z, 0, 8, 1e-5, z) == 1
    assert lib.logismos_launch_gemv_int4_g32_bf16(z, z, z, z, 1, 16, 100, z) == 1     # k % 128
    assert lib.logismos_launch_gemv_int4_g32_bf16(z, z, z, z, 65, 16, 128, z) == 1    # batch > 64
    assert lib.logismos_launch_linear_t_bf16(z, z, z, z, 8, 16, 100, 100, 16, 0, z, z) == 1  # k % 64
    assert lib.logismos_launch_varlen_attention_bf16(z, z, z, 1, 8, 4, 3, 128, 1024, 512, 768, 0, z) == 1  # heads % kv
    assert lib.logismos_launch_varlen_attention_bf16(z, z, z, 1, 8, 4, 2, 64, 512, 256, 384, 0, z) == 1    # head_dim
    assert lib.logismos_launch_varlen_attention_tc_bf16(z, z, z, z, 8, 1, 8, 4, 2, 64, 512, 256, 384, 0, z, z) == 1   # head_dim
    assert lib.logismos_launch_varlen_attention_tc_bf16(z, z, z, z, 8, 1, 8, 4, 3, 128, 1024, 512, 768, 0, z, z) == 1  # heads % kv, no scratch
    assert lib.logismos_varlen_attention_tc_scratch_bytes(100, 3, 2, 128) == 256 + 2 * 128 * 128 * 2  # 100 + 24 -> 128 padded keys
    assert lib.logismos_varlen_attention_tc_scratch_bytes(100, 3, 2, 64) == 0
    assert lib.logismos_launch_paged_attention_decode_bf16(z, z, z, z, z, z, z, z, z, z, z, 1, 1, 100, 4, 4, 16, 2, 128, z) == 1


def test_runtime_shim_returns_a_status_on_a_machine_without_a_gpu():
    """Every lg_* call must come back with a status (never spin or abort), device or not: on a box
    without a driver the calls fail with a classified code, on a GPU box they succeed."""
    n = C.c_int32(-1)
    rc = lib.lg_device_count(C.byref(n))
    assert (rc == 0 and n.value >= 1) or (rc != 0 and n.value == 0)
    d = C.c_void_p(123)
    rc = lib.lg_malloc(2**31 - 1, 64, C.byref(d))  # an ordinal no machine has: fails before allocating
    assert rc != 0 and d.value is None
    assert lib.lg_device_set_current(2**31 - 1) != 0
    s = C.c_void_p(77)
    assert lib.lg_stream_create(2**31 - 1, C.byref(s)) != 0 and s.value is None
    ms = C.c_float(0)
    assert lib.lg_event_elapsed_ms(None, None, None) == 1  # null out-pointer: InvalidValue


def test_error_kind_names_need_no_device():
    name = lambda c: lib.lg_error_kind_name(lib.lg_error_kind_from_raw(c)).decode()
    assert name(2) == "OutOfMemory" and name(700) == "IllegalAddress" and name(719) == "LaunchFailure"


def test_build_packing_matches_oracle_bit_for_bit():
    rng = np.random.default_rng(0)
    bs, n_pool, n = 16, 4096, 68
    cached = np.concatenate([rng.integers(256, 8193, 64), np.zeros(4)]).astype(np.int32)   # 64 decode + 4 prefill
    new = np.concatenate([np.ones(64), np.full(4, 512)]).astype(np.int32)
    need = -(-(cached + new) // bs)
    n_pool = int(need.sum()) + 5
    perm = rng.permutation(n_pool).astype(np.int32)
    tables = -np.ones((n, int(need.max()) + 1), np.int32); o = 0
    for i in range(n):
        tables[i, :need[i]] = perm[o:o + need[i]]; o += need[i]
    want = O.build_packing(cached, new, tables, bs, n_pool)
    total = int(new.sum())
    cu = np.empty(n + 1, np.int32); pos = np.empty(total, np.int32); slots = np.empty(total, np.int64); sid = np.empty(total, np.int32)
    P = lambda a: a.ctypes.data_as(C.c_void_p)
    r = lib.logismos_build_packing(P(cached), P(new), n, P(tables), tables.shape[1], bs, n_pool, P(cu), P(pos), P(slots), P(sid))
    assert r == total == 2112
    for got, ref in zip((cu, pos, slots, sid), want):
        assert (got == ref).all()
    tables[3, cached[3] // bs] = n_pool  # the block the new token of sequence 3 lands in: out of range -> rejected
    assert lib.logismos_build_packing(P(cached), P(new), n, P(tables), tables.shape[1], bs, n_pool, P(cu), P(pos), P(slots), P(sid)) == -1


def test_build_decode_chunks():
    cl = np.array([1, 512, 513, 17, 32768], np.int32); off = np.empty(6, np.int32)
    P = lambda a: a.ctypes.data_as(C.c_void_p)
    assert lib.logismos_build_decode_chunks(P(cl), 5, 512, P(off)) == 69
    assert off.tolist() == [0, 1, 2, 4, 5, 69]
    cl[3] = 0  # a context counts the token being decoded: an empty one is rejected
    assert lib.logismos_build_decode_chunks(P(cl), 5, 512, P(off)) == -1
    assert lib.logismos_paged_decode_scratch_bytes(68, 16, 128) == 68 * 16 * 130 * 4


def test_skinny_int4_route_table():
    """The kernel choice of logismos_launch_skinny_int4_g32_bf16 (host arithmetic): the tensor-core route above
    16 rows, for k >= 3 n at every batch, and from 8 rows up to n = 16384; the GEMV otherwise and whenever
    the shape rules of the tensor-core kernel do not hold."""
    want = {(1536, 1536, 1): 0, (1536, 1536, 8): 1, (1536, 1536, 16): 1, (1536, 1536, 64): 1, (8960, 1536, 4): 0, (8960, 1536, 16): 1,
            (1536, 8960, 1): 1, (1536, 8960, 64): 1, (151936, 1536, 1): 0, (151936, 1536, 16): 0, (151936, 1536, 17): 1,
            (17920, 1536, 16): 0, (2048, 6144, 2): 1, (256, 640, 64): 0, (1001, 1536, 40): 0, (1536, 1536, 65): 0, (1536, 1536, 0): 0}
    for (n, k, b), route in want.items():
        assert lib.logismos_skinny_int4_route(b, n, k) == route, (n, k, b)


def linear_tile(m, n, k, epilogue, sms=148):
    t = np.zeros(3, np.int32)
    assert lib.logismos_linear_t_tile(m, n, k, epilogue, None, sms, t.ctypes.data_as(C.c_void_p)) == 0
    return t.tolist()


def test_slices_of_k_only_where_half_the_sms_are_idle():
    """Slices of k meet in unordered reduce-adds, so the accumulating linear has them only where tiles of 128 x 128 leave at least
    half the SMs idle and k has eight blocks; every other output, and every other epilogue, is one sum."""
    for n in (256, 1000, 1536, 2048, 2560, 6144, 8960):
        for k in (64, 448, 512, 1536, 4096, 8960):
            for m in list(range(1, 1700, 37)) + [128, 129, 512, 513, 768, 769, 1024, 1025, 1152, 1153, 1536, 1537, 2929, 4096, 20384]:
                cols, pair, slices = linear_tile(m, n, k, 1)
                few = 2 * -(-m // 128) * -(-n // 128) <= 148 and k >= 512
                assert (slices > 1) <= few and cols in (128, 192, 256) and pair in (0, 1), (m, n, k, cols, pair, slices)
                assert slices == 1 or -(-m // 128) * -(-n // cols) * slices <= 148
                assert linear_tile(m, n, k, 0)[2] == 1
    assert linear_tile(768, 1536, 8960, 1)[2] > 1 and linear_tile(769, 1536, 8960, 1)[2] == 1 and linear_tile(513, 2048, 8192, 1)[2] == 1
    det = lib.logismos_get_deterministic()
    lib.logismos_set_deterministic(1)
    try:
        assert linear_tile(64, 1536, 8960, 1)[2] == 1
    finally:
        lib.logismos_set_deterministic(det)


def test_tile_of_a_linear_is_near_the_best_measured_one():
    """(rows, columns, k, epilogue) -> time in us of (columns, pair, slices), each timed alone on a B200; what is chosen takes at most 5 % more than the best.
    The shapes are those where an estimate without starts and without the reduce-adds of slices chose badly."""
    measured = {(300, 1536, 1536, 1): {(128, 0, 4): 6.24, (192, 0, 6): 6.58, (256, 0, 4): 7.9}, (400, 1536, 1536, 1): {(128, 0, 3): 6.97, (256, 0, 6): 7.37},
                (512, 1536, 1536, 1): {(128, 0, 3): 7.11, (192, 0, 4): 7.5, (256, 0, 6): 7.57}, (136, 2048, 2048, 1): {(128, 0, 4): 7.25, (256, 0, 8): 8.82},
                (200, 2048, 2048, 1): {(128, 0, 4): 7.00, (256, 0, 8): 8.67}, (2500, 1536, 2048, 0): {(256, 0, 1): 16.56, (256, 1, 1): 17.36},
                (2929, 1536, 2048, 0): {(256, 0, 1): 16.96, (256, 1, 1): 17.76}, (1200, 2048, 4096, 1): {(192, 0, 1): 28.04, (256, 1, 1): 29.22, (256, 0, 1): 30.1},
                (512, 1536, 8960, 1): {(256, 0, 6): 16.5, (128, 0, 3): 20.1, (192, 0, 4): 18.7}, (20384, 1536, 8960, 1): {(256, 1, 1): 399.0, (256, 0, 1): 446.0, (128, 0, 1): 714.0}}
    for (m, n, k, e), times in measured.items():
        got = tuple(linear_tile(m, n, k, e))
        assert times[got] <= 1.05 * min(times.values()), (m, n, k, got)


def test_process_wide_switches_and_scratch_sizes_need_no_device():
    assert lib.logismos_get_dependent_launch() in (0, 1)
    before = lib.logismos_get_dependent_launch()
    lib.logismos_set_dependent_launch(0); assert lib.logismos_get_dependent_launch() == 0
    lib.logismos_set_dependent_launch(1); assert lib.logismos_get_dependent_launch() == 1
    lib.logismos_set_dependent_launch(before)
    det = lib.logismos_get_deterministic()
    lib.logismos_set_deterministic(1); assert lib.logismos_get_deterministic() == 1
    lib.logismos_set_deterministic(det)
    # one slot of 57856 bytes per (64-token chunk, head); every sequence may end in a partial chunk
    assert lib.logismos_gdn_chunked_scratch_bytes(4096, 4, 16) == (64 + 4) * 16 * 57856
    assert lib.logismos_gdn_chunked_scratch_bytes(63, 1, 2) == 1 * 2 * 57856
    assert lib.logismos_gdn_chunked_scratch_bytes(-1, 1, 2) == 0 and lib.logismos_gdn_chunked_scratch_bytes(64, 1, 0) == 0
    assert lib.logismos_turbo3_row_bytes(256) == 112 and lib.logismos_turbo3_row_bytes(100) == 0


def test_python_ops_reject_cpu_operands_without_touching_a_device():  # praxis/src/matmul.rs:154-166
    import torch
    from logismos_b200 import ops
    a = torch.zeros((16, 16), dtype=torch.float16)
    with pytest.raises(ops.InvalidOp):
        ops.matmul(a, a)
    with pytest.raises(ops.InvalidOp):
        ops.softmax(a)


def test_rows_to_the_host_call_cuda_from_one_thread(tmp_path):
    """HostRows (logits to pageable memory) against a stand-in of the CUDA runtime: rows reach their places with and without pinned memory,
    errors come back, and the helper threads, which stand on device 0, make no CUDA call."""
    import os
    import subprocess
    here = os.path.dirname(os.path.abspath(__file__))
    root, exe = os.path.dirname(here), str(tmp_path / "host_rows")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "logismos_b200", "csrc"), "-I" + os.path.join(cuda, "include"),
                           os.path.join(here, "host_rows_check.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_layouts_of_the_one_launch_decode_step(tmp_path):
    """Every layout that stack_plan accepts: parts of shared memory that are live together lie apart, within the launch's bytes and aligned; every weight row has a CTA."""
    import os
    import subprocess
    here = os.path.dirname(os.path.abspath(__file__))
    root, exe = os.path.dirname(here), str(tmp_path / "decode_plan")
    csrc, cuda = os.path.join(root, "logismos_b200", "csrc"), os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + csrc, "-I" + os.path.join(cuda, "include"), os.path.join(here, "decode_plan_check.cpp"), os.path.join(csrc, "decode_plan.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_asynchronous_copies_and_barriers_are_ordered_for_the_compiler():
    """Inline instructions that start or await asynchronous copies, or that arrive at a barrier, say that they touch memory: without it the compiler may move plain accesses of the
    same shared memory across them."""
    import glob
    import os
    import re
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "logismos_b200", "csrc")
    seen = 0
    for path in sorted(glob.glob(os.path.join(csrc, "*.cu*")) + glob.glob(os.path.join(csrc, "*.h"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"\basm\b(?: volatile)?\s*\(", text):
            body = text[m.start():text.index(");", m.end())]
            if re.search(r"cp\.(reduce\.)?async|mbarrier\.|tcgen05\.(commit|mma)|barrier\.cluster", body):
                seen += 1
                assert '"memory"' in body, (os.path.basename(path), body)
    assert seen > 20
