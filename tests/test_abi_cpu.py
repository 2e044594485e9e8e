"""CPU-only checks: the C-ABI library loads and exports every symbol the header declares,
its GPU-free entry points behave, the host-side mirror's logic is right, and the committed
golden fixtures agree with the oracle."""
import ctypes as C
import re
from pathlib import Path

import numpy as np
import pytest

import oracle
from bitnet_mlx_rs_b200 import _lib as L
from bitnet_mlx_rs_b200 import cuda
from bitnet_mlx_rs_b200.bitlinear import absmean_quantize_weights

ROOT = Path(__file__).resolve().parents[1]
GOLDEN = ROOT / "tests" / "golden"


def declared_functions():
    names = []
    for h in (ROOT / "include").glob("*.h"):
        text = re.sub(r"/\*.*?\*/", "", h.read_text(), flags=re.S)
        names += re.findall(r"\b(bitnet_\w+|launch_w2a8_gemv_optimized)\s*\(", text)
    return sorted(set(names))


def test_library_exports_every_declared_symbol():
    lib = L.load()
    names = declared_functions()
    assert len(names) >= 30
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/ but not exported"
    # and the ctypes table covers exactly the header
    assert set(L.SIGNATURES) == set(names)


def test_status_strings_and_recoverability():
    lib = L.load()
    assert lib.bitnet_status_string(0) == b"ok"
    # bitnet-cuda/src/error.rs:88-103
    rec = {L.ERR_MEMORY_ALLOCATION, L.ERR_KERNEL_EXECUTION, L.ERR_STREAM_SYNC, L.ERR_PERFORMANCE, L.ERR_CUDA_DRIVER}
    non = {L.ERR_CUDA_NOT_ENABLED, L.ERR_DEVICE, L.ERR_INVALID_CONFIG, L.ERR_UNSUPPORTED_OPERATION,
           L.ERR_UNSUPPORTED_DTYPE, L.ERR_INCOMPATIBLE_SHAPES}
    for s in rec:
        assert lib.bitnet_is_recoverable(s) == 1
    for s in non:
        assert lib.bitnet_is_recoverable(s) == 0
    assert cuda.IncompatibleShapes("x").is_recoverable() is False
    assert cuda.MemoryAllocation("x").is_recoverable() is True


def test_config_defaults_match_reference():
    cfg = L.BackendConfig()
    L.load().bitnet_backend_config_default(C.byref(cfg))
    # bitnet-cuda/src/backend.rs:27-37 and kernels/w2a8_gemv.rs:28-38
    assert (cfg.device_id, cfg.memory_pool_size, cfg.num_streams, cfg.enable_profiling) == (0, 1 << 30, 4, 0)
    w = cfg.w2a8_config
    assert (w.block_size, w.grid_strategy, w.enable_weight_permutation, w.enable_dp4a, w.coalescing_level) == \
        (256, 1, 1, 1, 2)
    d = cuda.CudaBackendConfig()
    assert (d.device_id, d.memory_pool_size, d.num_streams) == (0, 1 << 30, 4)
    assert cuda.MEMORY_BANDWIDTH_TARGET == 85.0 and cuda.W2A8_SPEEDUP_MAX == 3.63


def test_argument_errors_need_no_gpu():
    lib = L.load()
    assert lib.bitnet_bitlinear_forward(None, 1.0, None, None, 4, 64, 64, None, None, 0, None) == L.ERR_NULL_POINTER
    assert b"null" in lib.bitnet_last_error_string()
    assert lib.bitnet_bitlinear_forward(None, 1.0, None, None, 0, 64, 64, None, None, 0, None) == L.OK   # empty batch
    assert lib.bitnet_w2a8_gemv(None, None, None, 0, 64, None) == L.OK
    assert lib.bitnet_w2a8_gemv(None, None, None, 8, 64, None) == L.ERR_NULL_POINTER
    assert lib.bitnet_w2a8_gemv(1, 1, 1, 8, 0, None) == L.ERR_INCOMPATIBLE_SHAPES
    assert lib.bitnet_quantize_activations(1, 2, 0, 1, 1, None) == L.ERR_INCOMPATIBLE_SHAPES
    n = C.c_size_t(123)
    # decode path: room for the once-quantised activations (int8, fragment order) of 8 tokens
    assert lib.bitnet_bitlinear_workspace_size(8, 2560, 6912, L.PATH_AUTO, C.byref(n)) == L.OK
    assert 8 * 2560 <= n.value <= 64 * 1024 and n.value % 256 == 0
    assert lib.bitnet_bitlinear_workspace_size(3, 37, 29, L.PATH_AUTO, C.byref(n)) == L.OK and n.value >= 3 * 37 + 12
    assert lib.bitnet_bitlinear_workspace_size(8, 64, 64, 99, C.byref(n)) == L.ERR_INVALID_CONFIG
    with pytest.raises(cuda.NullPointer):
        cuda.check(L.ERR_NULL_POINTER)


def test_backend_without_gpu_reports_cuda_not_enabled():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    assert cuda.is_cuda_available() is False
    with pytest.raises(cuda.CudaNotEnabled):
        cuda.CudaBackend()


def test_host_absmean_quantiser_matches_oracle():
    rng = np.random.default_rng(1)
    w = rng.standard_normal((96, 160)).astype(np.float32)
    qw = absmean_quantize_weights(w)
    t, scale = oracle.absmean_quantize_weights(w)
    assert np.array_equal(qw.values, t)
    assert qw.scale == pytest.approx(scale, rel=1e-6)
    assert absmean_quantize_weights(np.zeros((4, 4), np.float32)).scale == 1.0   # weights.rs:554-556


@pytest.mark.parametrize("path", sorted(GOLDEN.glob("*.npz")), ids=lambda p: p.stem)
def test_oracle_reproduces_golden_fixtures(path):
    z = np.load(path)
    if "gate" in z:
        y, h = oracle.ffn_forward(z["gate"], float(z["s_gate"]), z["up"], float(z["s_up"]), z["down"],
                                  float(z["s_down"]), z["x"], int(z["ffn"]))
        assert np.array_equal(y, z["y"]) and np.array_equal(h, z["h"])
        return
    ref = oracle.bitlinear_forward(z["wp"], float(z["w_scale"]), z["x"], int(z["N"]))
    for key in ("q", "acc", "a_scale", "y"):
        assert np.array_equal(ref[key], z[key]), key


def test_stack_block_follows_its_values():
    """Scales may be objects that change between calls (0-d tensors, arrays): the block holds what they hold now."""
    import torch

    from bitnet_mlx_rs_b200 import ops

    def block(rows, scales):
        return L.Stack.from_buffer_copy(ops._stack(rows, scales))

    for cell in (torch.tensor(0.5), np.array(0.5)):
        assert list(block([64, 32], [cell, 0.25]).scales) == [0.5, 0.25, 0.0]
        cell.fill_(9.0) if torch.is_tensor(cell) else cell.fill(9.0)
        assert list(block([64, 32], [cell, 0.25]).scales) == [9.0, 0.25, 0.0]
    st = block((np.int64(64), torch.tensor(32), 8), (1, np.float32(2.5), -0.0))
    assert (st.n_members, list(st.rows)) == (3, [64, 32, 8])
    assert list(st.scales) == [1.0, 2.5, 0.0] and np.signbit(st.scales[2]) and not np.signbit(block((64, 32, 8), (1, 2.5, 0.0)).scales[2])
    assert list(block([64], [1e39]).scales)[0] == float("inf") and list(block([64, 1], [2.0]).scales) == [2.0, 0.0, 0.0]
    assert all(p.size == C.sizeof(L.Stack) for p in ops._STACKS.values())
    for rows, scales in (([64.0], [1.0]), ([64], ["1"]), ([1, 2, 3, 4], [1.0])):
        with pytest.raises((TypeError, IndexError)):
            ops._stack(rows, scales)


@pytest.mark.parametrize("hidden,ffn", [(256, 192), (192, 256), (256, 1000)])
@pytest.mark.parametrize("M", [4, 40, 200])
def test_ffn_by_a_named_path_refuses_widths_the_path_does_not_take(M, hidden, ffn):
    """Refused before anything is launched: the addresses are never used."""
    lib, opts = L.load(), L.ForwardOpts(path=L.PATH_PREFILL)
    args = (M, hidden, ffn, C.byref(opts), 1 << 20, 1 << 40, None)
    for fn, glue in ((lib.bitnet_ffn_forward, ()), (lib.bitnet_ffn_forward_fused, (None,))):
        st = fn(4096, 0.1, 4096, 0.1, 4096, 0.1, 4096, *glue, 4096, 4096, *args)
        assert st == L.ERR_UNSUPPORTED_OPERATION, lib.bitnet_last_error_string()


@pytest.mark.parametrize("M,K,N", [(9, 8320, 256), (16, 8320, 32768), (17, 2560, 640), (128, 2560, 2560)])
def test_auto_refuses_peer_outputs_where_the_cluster_kernel_was_its_choice(M, K, N):
    opts = L.ForwardOpts(n_peers=1)
    opts.y_peers_dev[0] = 4096
    st = L.load().bitnet_bitlinear_forward(4096, 0.1, 4096, 4096, M, K, N, C.byref(opts), 1 << 20, 1 << 40, None)
    assert st == L.ERR_UNSUPPORTED_OPERATION


@pytest.mark.parametrize("K,off,status", [(1002, 0, "ERR_UNSUPPORTED_OPERATION"), (3000, 0, "ERR_UNSUPPORTED_OPERATION"), (16400, 0, "ERR_UNSUPPORTED_OPERATION"),
                                          (1040, 4, "ERR_INVALID_CONFIG"), (2576, 1, "ERR_INVALID_CONFIG")])
def test_glue_that_no_kernel_takes_is_refused_before_anything_runs(K, off, status):
    """Odd widths with row glue: the addresses are never used."""
    lib, M, N = L.load(), 40, 3000
    glue = L.RowGlue(4096 + off, None, None, None, 1e-5, None)
    stack = L.Stack(1, (C.c_size_t * 3)(N), (C.c_float * 3)(0.1))
    st = lib.bitnet_bitlinear_forward_fused(4096, C.byref(stack), 4096, C.byref(glue), 4096, M, K, None, 1 << 20, 1 << 40, None)
    assert st == getattr(L, status), lib.bitnet_last_error_string()
