"""The C-ABI library without a GPU: it loads, exports every symbol the header
declares, and rejects bad arguments with an error code before touching CUDA."""
import ctypes as C
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared():
    text = open(os.path.join(ROOT, "include", "lmoe.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(lmoe_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_exported():
    from maxuna_b200 import _native

    lib = _native.lib()
    names = _declared()
    assert len(names) >= 25
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/lmoe.h but not exported"
    assert set(names) == set(_native.PROTOTYPES), set(names) ^ set(_native.PROTOTYPES)
    assert b"sm_100a" in lib.lmoe_version()


def test_ffn_mm_width_limit_is_the_headers():
    from maxuna_b200 import ops

    text = open(os.path.join(ROOT, "include", "lmoe.h")).read()
    assert ops.FFN_MM_MAX_FF == int(re.search(r"#define LMOE_FFN_MM_MAX_FF (\d+)", text).group(1))


def test_argument_errors_without_cuda():
    from maxuna_b200 import _native

    lib = _native.lib()
    h = C.c_void_p()
    # bad dtype, bad k, size mismatch, misaligned base_off: errors, not crashes
    assert lib.lmoe_expert_stack_wrap(99, 1, 8, 256, 16, 8 * 144, 0, C.byref(h)) == -1
    assert b"dtype" in lib.lmoe_last_error()
    assert lib.lmoe_expert_stack_wrap(12, 1, 8, 100, 16, 8 * 144, 0, C.byref(h)) == -1
    assert b"multiple" in lib.lmoe_last_error()
    assert lib.lmoe_expert_stack_wrap(12, 1, 8, 256, 16, 7 * 144, 0, C.byref(h)) == -1
    assert lib.lmoe_expert_stack_wrap(12, 1, 8, 256, 16, 8 * 144, 8, C.byref(h)) == -1
    assert lib.lmoe_expert_stack_wrap(12, 4, 8, 256, 4096, 4 * 8 * 144, 0, C.byref(h)) == 0
    # mul_mv_id seam checks (src/ops/dispatch.rs:812-847 of the reference)
    fake = C.c_void_p(4096)
    assert lib.lmoe_mul_mv_id(h, fake, 1, 1, 128, fake, 1, 2, fake, None) == -1
    assert b"does not match expert stack k" in lib.lmoe_last_error()
    assert lib.lmoe_mul_mv_id(h, fake, 2, 1, 256, fake, 3, 2, fake, None) == -1
    assert b"ids t" in lib.lmoe_last_error()
    assert lib.lmoe_mul_mv_id(h, fake, 2, 3, 256, fake, 2, 2, fake, None) == -1
    assert b"x_per_row" in lib.lmoe_last_error()
    lib.lmoe_expert_stack_destroy(h)
    # combine guards (src/ops/dispatch.rs:294-305)
    assert lib.lmoe_combine(fake, None, fake, 1, 130, 8, fake, None) == -1
    assert lib.lmoe_combine(fake, None, fake, 1 << 20, 10, 3072, fake, None) == -1
    assert b"i32::MAX" in lib.lmoe_last_error()
    # routing guards
    assert lib.lmoe_route_from_logits(fake, None, 1, 1000, 10, 2.5, 1, fake, fake, None) == -1
    assert lib.lmoe_route_from_logits(fake, None, 1, 8, 9, 2.5, 1, fake, fake, None) == -1
    # workspace guard
    assert lib.lmoe_prepare_map0(fake, 16, 2, 4, fake, 8, None) == -4
    assert lib.lmoe_map0_scratch_bytes(256, 512) >= 256 * 4 + 256 * 512 * 4


def test_ffn_mm_argument_errors_without_cuda():
    from maxuna_b200 import _native

    lib = _native.lib()
    fake, keep = C.c_void_p(4096), []

    def stack(ne, n_out, k, dt=12):
        h = C.c_void_p()
        assert lib.lmoe_expert_stack_wrap(dt, ne, n_out, k, 4096, ne * n_out * k // 256 * (144 if dt == 12 else 210), 0, C.byref(h)) == 0
        keep.append(h)
        return h

    def call(g, u, d, t=4, t_ids=4, top_k=2, k=512, ids=fake, w=fake, x=fake, ws=fake, n=None, out=fake):
        n = lib.lmoe_ffn_mm_workspace_bytes(g, d, t, top_k) if n is None else n
        return lib.lmoe_ffn_mm(g, u, d, ids, t_ids, top_k, w, x, t, k, out, ws, n, None)

    g, u, d = stack(4, 256, 512), stack(4, 256, 512), stack(4, 512, 256, 14)
    need = lib.lmoe_ffn_mm_workspace_bytes(g, d, 4, 2)
    assert need > 0 and lib.lmoe_ffn_mm_workspace_bytes(g, None, 4, 2) == 0 and lib.lmoe_ffn_mm_workspace_bytes(g, d, -1, 2) == 0
    for bad in (dict(k=256), dict(t_ids=3), dict(ids=None), dict(w=None), dict(x=None), dict(out=None), dict(x=C.c_void_p(4100)), dict(top_k=0)):
        assert call(g, u, d, **bad) == -1, bad
    # stacks that disagree: widths, numbers of experts, the down product's k
    assert call(g, stack(4, 128, 512), d) == -1
    assert call(g, stack(3, 256, 512), d) == -1 and b"disagree" in lib.lmoe_last_error()
    assert call(g, u, stack(3, 512, 256, 14)) == -1 and b"disagree" in lib.lmoe_last_error()
    assert call(g, u, stack(4, 512, 512, 14)) == -1
    assert call(g, None, d) == -1
    # more activations than the separate silu_mul takes
    assert call(g, u, d, t=1 << 22, t_ids=1 << 22) == -1 and b"i32::MAX" in lib.lmoe_last_error()
    # workspace: missing, a byte short, not on 256 bytes
    assert call(g, u, d, ws=None) == -4 and call(g, u, d, n=need - 1) == -4 and call(g, u, d, ws=C.c_void_p(4096 + 128)) == -4
    # a row that does not fit into shared memory: the ops one by one take it
    assert call(stack(1, 12544, 512), stack(1, 12544, 512), stack(1, 512, 12544, 14)) == -2 and b"one by one" in lib.lmoe_last_error()
    for h in keep:
        lib.lmoe_expert_stack_destroy(h)


def test_expert_parallel_argument_errors_without_cuda():
    from maxuna_b200 import _native

    lib = _native.lib()
    fake = C.c_void_p(4096)
    # n_expert must divide over the ranks, hidden a multiple of 8, buffers non-NULL and aligned
    assert lib.lmoe_ep_pack(fake, fake, fake, 4, 128, 2, 8, 3, fake, fake, fake, fake, fake, fake, 1 << 20, None) == -1
    assert b"divisible" in lib.lmoe_last_error()
    assert lib.lmoe_ep_pack(fake, fake, fake, 4, 100, 2, 8, 2, fake, fake, fake, fake, fake, fake, 1 << 20, None) == -1
    assert lib.lmoe_ep_pack(fake, fake, fake, 4, 128, 2, 8, 2, None, fake, fake, fake, fake, fake, 1 << 20, None) == -1
    assert lib.lmoe_ep_pack(C.c_void_p(4100), fake, fake, 4, 128, 2, 8, 2, fake, fake, fake, fake, fake, fake, 1 << 20, None) == -1
    assert b"aligned" in lib.lmoe_last_error()
    assert lib.lmoe_ep_pack(fake, fake, fake, 4, 128, 2, 8, 2, fake, fake, fake, fake, fake, fake, 16, None) == -4
    assert lib.lmoe_ep_pack_workspace_bytes(8, 4) >= 8 * 4 + 8 * 4 * 4
    assert lib.lmoe_ep_combine(None, fake, None, 4, 2, 128, fake, None) == -1
    assert lib.lmoe_ep_combine(fake, fake, None, 4, 0, 128, fake, None) == -1
    assert lib.lmoe_ep_combine(fake, fake, None, 0, 2, 128, fake, None) == 0
    assert lib.lmoe_experts_forward_rows_f16(None, fake, fake, fake, 4, fake, fake, 1 << 20, None) == -1


def test_peer_and_host_entry_argument_errors_without_cuda():
    """The peer-memory exchange and the host-buffer entries check their arguments before they touch the GPU."""
    from maxuna_b200 import _native

    lib = _native.lib()
    fake = C.c_void_p(4096)
    arr = (C.c_void_p * 2)(4096, 8192)
    assert lib.lmoe_peer_ctrl_bytes() >= 128 * 4
    assert lib.lmoe_peer_alloc(0, C.byref(C.c_void_p()), C.create_string_buffer(64)) == -1
    assert lib.lmoe_peer_open(None, C.byref(C.c_void_p())) == -1
    assert lib.lmoe_peer_put(None, 64, 2, 0, 0, arr, arr, fake, 0, None) == -1
    assert lib.lmoe_peer_put(fake, 64, 17, 0, 0, arr, arr, fake, 0, None) == -1          # more ranks than the kernel carries
    assert lib.lmoe_peer_put(fake, 64, 2, 2, 0, arr, arr, fake, 0, None) == -1           # rank outside the world
    assert lib.lmoe_peer_put(fake, 40, 2, 0, 0, arr, arr, fake, 0, None) == -1           # chunk not a multiple of 16
    assert b"16" in lib.lmoe_last_error()
    assert lib.lmoe_peer_put(fake, 64, 2, 0, 0, arr, arr, fake, 2, None) == -1           # direction is 0 or 1
    assert lib.lmoe_peer_wait(None, 2, 0, None) == -1
    assert lib.lmoe_peer_wait(fake, 0, 0, None) == -1
    for fn in (lib.lmoe_moe_forward_host, lib.lmoe_moe_forward_host_async):
        assert fn(None, fake, 1, fake, None, None, fake, 1 << 20, None) == -1
        assert b"layer" in lib.lmoe_last_error()


def test_host_mirror_rejects_cpu_tensors():
    import torch

    from maxuna_b200 import LmoeError, ops

    with pytest.raises(LmoeError):
        ops.silu_mul(torch.zeros(4), torch.zeros(4))
    with pytest.raises(LmoeError):
        ops.combine(torch.zeros(1, 2, 3), None, torch.zeros(1, 2))


def test_cpp_host_mirror_compiles_and_reports_errors(tmp_path):
    import shutil
    import subprocess

    from maxuna_b200 import _native

    _native.lib()
    gxx = shutil.which("g++")
    assert gxx, "g++ not found"
    exe = str(tmp_path / "host_errors")
    libdir = os.path.dirname(_native.lib_path())
    env = {k: v for k, v in os.environ.items() if k not in ("CC", "CXX")}
    subprocess.run([gxx, "-std=c++17", "-O1", os.path.join(ROOT, "tests", "cpp", "host_errors.cpp"), "-o", exe,
                    "-L" + libdir, "-llmoe", "-Wl,-rpath," + libdir], check=True, env=env)
    out = subprocess.run([exe], capture_output=True, text=True, env=env)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
