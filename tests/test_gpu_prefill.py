"""Parity of the tensor-core (prefill) path with the CPU oracle, through the C ABI.
int8 activations, scales and int32 accumulators bit-exact; fp32 outputs within 1e-5 relative."""
from pathlib import Path

import numpy as np
import pytest
import torch

import oracle
from bitnet_mlx_rs_b200 import ops

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"
RTOL = 1e-5


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def case(seed, M, K, N):
    return oracle.gen_ternary_packed(seed, 1, N * K), oracle.gen_weight_scale(seed, 1, K), oracle.gen_activations(seed, 2, (M, K))


@pytest.mark.parametrize("M,K,N", [(128, 128, 256), (256, 256, 128), (1, 128, 8), (130, 384, 700), (300, 1024, 513),
                                   (17, 2560, 640), (512, 640, 2560)])
def test_prefill_matches_oracle(M, K, N):
    wp, ws, x = case(500 + M, M, K, N)
    ref = oracle.bitlinear_forward(wp, ws, x, N)
    y, dbg = ops.bitlinear_forward(dev(wp), ws, dev(x), N, debug=True, path="prefill")
    assert ops.device_error_flags() == 0
    assert np.array_equal(dbg["q"].cpu().numpy(), ref["q"])
    assert np.array_equal(dbg["a_scale"].cpu().numpy(), ref["a_scale"])
    assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
    np.testing.assert_allclose(y.cpu().numpy(), ref["y"], rtol=RTOL, atol=0)
    assert np.array_equal(y.cpu().numpy(), ref["y"])


def test_prefill_golden_fixture():
    z = np.load(GOLDEN / "prefill_m256_k256_n128.npz")
    y, dbg = ops.bitlinear_forward(dev(z["wp"]), float(z["w_scale"]), dev(z["x"]), int(z["N"]), debug=True, path="prefill")
    assert np.array_equal(dbg["acc"].cpu().numpy(), z["acc"])
    np.testing.assert_allclose(y.cpu().numpy(), z["y"], rtol=RTOL, atol=0)


def test_auto_dispatch_uses_tensor_cores_for_many_tokens():
    M, K, N = 200, 256, 96
    wp, ws, x = case(9, M, K, N)
    y = ops.bitlinear_forward(dev(wp), ws, dev(x), N)
    assert np.array_equal(y.cpu().numpy(), oracle.bitlinear_forward(wp, ws, x, N)["y"])


@pytest.mark.parametrize("K,N", [(2560, 2560), (2560, 640), (2560, 6912), (6912, 2560)])
def test_prefill_layer_shapes_at_2048_tokens(K, N):
    # one projection of the 2B decoder layer at M = 2048: the oracle checks sampled token rows against
    # sampled feature rows exactly; the decode kernel (already checked against the oracle) cross-checks
    # a block of 16 tokens on all features; a checksum identity covers everything else
    M = 2048
    wp, ws, x = case(600 + N // 64 + K // 64, M, K, N)
    dwp, dx = dev(wp), dev(x)
    y, dbg = ops.bitlinear_forward(dwp, ws, dx, N, debug=True, path="prefill")
    assert ops.device_error_flags() == 0
    rows = [0, 1, 127, 128, 1000, 2047]
    for f0 in (0, N // 2 - 32, N - 64):
        sl = wp[f0 * K // 4:(f0 + 64) * K // 4]
        ref = oracle.bitlinear_forward(sl, ws, x[rows], 64)
        assert np.array_equal(dbg["acc"][rows][:, f0:f0 + 64].cpu().numpy(), ref["acc"])
        np.testing.assert_allclose(y[rows][:, f0:f0 + 64].cpu().numpy(), ref["y"], rtol=RTOL, atol=0)
    y16, d16 = ops.bitlinear_forward(dwp, ws, dx[512:528].contiguous(), N, debug=True, path="decode")
    assert torch.equal(d16["acc"], dbg["acc"][512:528])
    assert torch.equal(y16, y[512:528])
    w = ops.unpack_ternary(dwp, N * K).reshape(N, K)
    colsum = w.sum(dim=0, dtype=torch.float64)
    assert torch.equal(dbg["acc"].sum(dim=1, dtype=torch.float64), dbg["q"].to(torch.float64) @ colsum)


@pytest.mark.gpu
@pytest.mark.parametrize("env", [{"BITNET_PREFILL_WHOLE": "0"}, {"BITNET_PREFILL_WHOLE": "0", "BITNET_PREFILL_BT": "64"},
                                 {"BITNET_PREFILL_WHOLE": "1", "BITNET_PREFILL_BT": "96"}])
def test_prefill_every_work_split(env):
    """The planner's other modes (tiles split between CTAs with the integer fix-up, smaller token
    tiles) give the same bits as the generic kernel.  The mode is read once per process, so each
    case runs in a child process."""
    import os
    import subprocess
    import sys
    code = r'''
import sys, torch
sys.path.insert(0, ".")
from bitnet_mlx_rs_b200 import ops
g = torch.Generator(device="cuda").manual_seed(5)
for (M, K, N) in [(2048, 2560, 640), (300, 1024, 384), (1000, 6912, 2560), (17, 128, 1), (256, 8192, 1024)]:
    w = torch.randint(0, 256, (N * K // 4,), dtype=torch.uint8, device="cuda", generator=g)
    ops.sanitize_packed(w)
    x = torch.randn(M, K, device="cuda", generator=g)
    y = ops.bitlinear_forward(w, 0.02, x, N, path="prefill")
    ref = ops.bitlinear_forward(w, 0.02, x, N, path="generic")
    assert torch.equal(y, ref), (M, K, N)
assert ops.device_error_flags() == 0
print("ok")
'''
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, **env), capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0 and "ok" in out.stdout, out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("ldy_extra,col0", [(64, 0), (64, 32), (3, 0), (5, 1)])
def test_prefill_strided_and_unaligned_output(ldy_extra, col0):
    """y with a row stride larger than N (a column slice of a wider output): rows that are
    16-byte aligned leave through TMA stores, anything else through plain stores; bytes outside
    the slice stay untouched."""
    M, K, N = 200, 512, 320
    g = torch.Generator(device="cuda").manual_seed(11)
    w = torch.randint(0, 256, (N * K // 4,), dtype=torch.uint8, device="cuda", generator=g)
    ops.sanitize_packed(w)
    x = torch.randn(M, K, device="cuda", generator=g)
    ref = ops.bitlinear_forward(w, 0.03, x, N, path="generic")
    ldy = N + ldy_extra
    wide = torch.full((M, ldy), -7.0, device="cuda")
    view = wide.view(-1)[col0:]           # the slice's first element
    ops.bitlinear_forward(w, 0.03, x, N, path="prefill", out=view, ldy=ldy)
    torch.cuda.synchronize()
    got = wide[:, col0:col0 + N]
    assert torch.equal(got, ref)
    mask = torch.ones_like(wide, dtype=torch.bool)
    mask[:, col0:col0 + N] = False
    assert bool((wide[mask] == -7.0).all())
    assert ops.device_error_flags() == 0


# ---- gate/up pair, stacked members, small calls ----------------------------------------------------------------

def _weights(g, n, k):
    w = torch.randint(0, 256, ((n * k + 3) // 4,), dtype=torch.uint8, device="cuda", generator=g)
    ops.sanitize_packed(w)
    return w


@pytest.mark.gpu
@pytest.mark.parametrize("M,H,F", [
    (17, 128, 132),       # one k slice, the last feature tile nearly empty
    (65, 384, 1000),      # an odd number of slices, both halves on CTAs of their own
    (200, 256, 20000),    # more tiles than SMs: a CTA takes several in turn (the pair is never split between CTAs)
    (33, 512, 130),       # rows of h that TMA cannot store (plain stores)
    (700, 2560, 640),
])
def test_gate_up_pair_matches_the_generic_kernels(M, H, F):
    """Integer sums and the same three fp32 multiplications: every bit agrees."""
    g = torch.Generator(device="cuda").manual_seed(M)
    wg, wu, wd = _weights(g, F, H), _weights(g, F, H), _weights(g, H, F)
    x = torch.randn(M, H, device="cuda", generator=g)
    x[M // 2] = 0.0       # an all-zero token
    ry, rh = ops.ffn_forward(wg, 0.05, wu, 0.04, wd, 0.03, x, F, path="generic")
    for _ in range(2):    # again over what the first call left in the workspace
        y, h = ops.ffn_forward(wg, 0.05, wu, 0.04, wd, 0.03, x, F)
        assert torch.equal(h, rh) and torch.equal(y, ry)
    assert ops.device_error_flags() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,rows", [(20, 256, (128, 64, 64)), (130, 384, (200, 56, 8)), (300, 1024, (1, 300)), (1000, 2560, (2560, 640, 640)),
                                      (2, 1024, (30000, 3000)), (12, 512, (20000, 10000, 77)),
                                      (149, 4096, (128, 64, 64)), (150, 5120, (64, 10)), (160, 8192, (128,)), (149, 128, (64,)), (150, 16384, (64,)),
                                      # tiles split between CTAs: both quantisers that clear the tiles' counters
                                      (200, 8192, (9000, 600, 100)), (140, 8192, (19000,))])
def test_stacked_members_with_glue_match_the_generic_kernels(M, K, rows):
    g = torch.Generator(device="cuda").manual_seed(M)
    w = _weights(g, sum(rows), K)
    x, res = torch.randn(M, K, device="cuda", generator=g), torch.randn(M, K, device="cuda", generator=g)
    nw, nb = torch.randn(K, device="cuda", generator=g), torch.randn(K, device="cuda", generator=g)
    scales = [0.05, 0.07, 0.02][:len(rows)]
    out = {}
    for path in ("generic", "prefill", "auto"):
        s, n = torch.empty_like(x), torch.empty_like(x)
        glue = ops.make_glue(residual=res, sum_out=s, norm_weight=nw, norm_bias=nb, eps=1e-5, normed_out=n)
        y, dbg = ops.bitlinear_forward_fused(w, rows, scales, x, glue=glue, path=path, debug=True)
        out[path] = (y, s, n, dbg["q"], dbg["a_scale"], dbg["acc"])
    for path in ("auto", "prefill"):
        for a, b in zip(out[path], out["generic"]):
            assert torch.equal(a, b), path
    assert ops.device_error_flags() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", [(2, 1024, 32768), (9, 4096, 11008), (16, 256, 80001), (8, 128, 60000),     # AUTO leaves the decode kernel
                                   (8, 2560, 60000), (16, 128, 40001)])                                       # and stays
def test_small_calls_on_either_kernel(M, K, N):
    """Shapes on both sides of the line between the two kernels: the same bits from both, and without a workspace."""
    import ctypes as C
    from bitnet_mlx_rs_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(M)
    w, x = _weights(g, N, K), torch.randn(M, K, device="cuda", generator=g)
    ref = ops.bitlinear_forward(w, 0.02, x, N, path="decode")
    assert torch.equal(ops.bitlinear_forward(w, 0.02, x, N), ref)
    y = torch.empty_like(ref)
    opts = L.ForwardOpts()
    st = L.load().bitnet_bitlinear_forward(w.data_ptr(), 0.02, x.data_ptr(), y.data_ptr(), M, K, N, C.byref(opts), None, 0,
                                           torch.cuda.current_stream().cuda_stream)
    assert st == 0 and torch.equal(y, ref)
    assert ops.device_error_flags() == 0


# ---- widths that are no multiple of 128 ------------------------------------------------------------------------

@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", [
    (17, 64, 50), (100, 8640, 320), (200, 192, 300), (2048, 320, 130),            # multiples of 64: half of the last slice is empty
    (1, 1001, 2100), (9, 333, 5000), (40, 1000, 600), (130, 130, 5000),           # rows that start in the middle of a byte
    (40, 8192, 640), (32, 4096, 1100), (33, 4096, 1100), (65, 8192, 2560),          # either side of the line to the cluster kernel
    (33, 4, 40000), (3, 65, 20001), (16, 16400, 140), (300, 2576, 77),            # (short rows stay on the generic kernel), wide, no multiple of 4 rows
    (700, 4, 4000), (40, 65, 20001), (90, 129, 333), (60, 127, 1001),             # one slice, one code past half a slice, past and short of a slice
    (200, 8256, 9700), (200, 8200, 9700),                                         # tiles split between CTAs, the last slice partly empty
])
def test_any_width_matches_the_generic_kernel(M, K, N):
    g = torch.Generator(device="cuda").manual_seed(K)
    w = _weights(g, N, K)
    x = torch.randn(M, K, device="cuda", generator=g)
    x[0] = 0.0
    y, d = ops.bitlinear_forward(w, 0.02, x, N, debug=True)
    ry, rd = ops.bitlinear_forward(w, 0.02, x, N, debug=True, path="generic")
    assert torch.equal(y, ry) and all(torch.equal(d[k], rd[k]) for k in rd)
    assert ops.device_error_flags() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,N", [(8, 1001, 2100), (40, 1001, 6000), (300, 2577, 3000)])
@pytest.mark.parametrize("glue", [False, True])
def test_odd_width_in_a_chain_of_programmatic_launches(M, K, N, glue):
    """Two matrices take turns on one workspace, every launch with programmatic start: the GEMM must read the rows that its own
    call copied to slice boundaries, not the other matrix's from the call before."""
    if glue:
        K = K // 16 * 16 + 16        # the glue takes multiples of 16; none of these is one of 64
    g = torch.Generator(device="cuda").manual_seed(N)
    ws, x = [_weights(g, N, K) for _ in range(2)], torch.randn(M, K, device="cuda", generator=g)
    nw, nb = torch.ones(K, device="cuda"), torch.zeros(K, device="cuda")      # (the glue holds addresses, not tensors)
    row_glue = ops.make_glue(residual=x, norm_weight=nw, norm_bias=nb)

    def call(w, **kw):
        return ops.bitlinear_forward_fused(w, (N,), (0.02,), x, glue=row_glue, **kw) if glue else ops.bitlinear_forward(w, 0.02, x, N, **kw)

    ref = [call(w, path="generic") for w in ws]
    out = [call(ws[i % 2], pdl=True) for i in range(20)]
    assert all(torch.equal(y, ref[i % 2]) for i, y in enumerate(out))
    assert ops.device_error_flags() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1002, 8640])
def test_any_width_any_alignment_and_workspace(K):
    """Buffers that start anywhere, code 3 (weight 0 to the generic kernel) and a workspace that only suits the generic kernel."""
    import ctypes as C
    from bitnet_mlx_rs_b200 import _lib as L
    M, N = 40, 700
    g = torch.Generator(device="cuda").manual_seed(K)
    nb = (N * K + 3) // 4
    store, xs = torch.randint(0, 256, (nb + 64,), dtype=torch.uint8, device="cuda", generator=g), torch.randn(M * K + 8, device="cuda", generator=g)
    if K % 64 == 0:
        ops.sanitize_packed(store)
    lib, opts = L.load(), L.ForwardOpts()
    need, least = C.c_size_t(), C.c_size_t()
    assert lib.bitnet_bitlinear_workspace_size(M, K, N, L.PATH_AUTO, C.byref(need)) == 0
    assert lib.bitnet_bitlinear_workspace_size(M, K, N, L.PATH_GENERIC, C.byref(least)) == 0
    ws = torch.empty(need.value + 256, dtype=torch.uint8, device="cuda")
    base = (ws.data_ptr() + 255) // 256 * 256
    stream = torch.cuda.current_stream().cuda_stream
    for w_off, x_off, size in ((0, 0, need.value), (1, 0, need.value), (4, 1, need.value), (16, 3, need.value), (0, 0, least.value)):
        out = []
        for path, nbytes in ((L.PATH_AUTO, size), (L.PATH_GENERIC, least.value)):
            opts.path = path
            y = torch.full((M, N), float("nan"), device="cuda")
            st = lib.bitnet_bitlinear_forward(store.data_ptr() + w_off, 0.02, xs.data_ptr() + 4 * x_off, y.data_ptr(), M, K, N, C.byref(opts),
                                              base, nbytes, stream)
            assert st == 0
            out.append(y)
        assert torch.equal(*out), (w_off, x_off, size)
    assert ops.device_error_flags() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,H,F", [(40, 192, 320), (40, 1000, 1500), (20, 2560, 1000), (5, 1000, 2560), (140, 320, 64)])
def test_ffn_of_any_width_matches_the_generic_kernels(M, H, F):
    g = torch.Generator(device="cuda").manual_seed(F)
    wg, wu, wd = _weights(g, F, H), _weights(g, F, H), _weights(g, H, F)
    x = torch.randn(M, H, device="cuda", generator=g)
    y, h = ops.ffn_forward(wg, 0.05, wu, 0.04, wd, 0.03, x, F)
    ry, rh = ops.ffn_forward(wg, 0.05, wu, 0.04, wd, 0.03, x, F, path="generic")
    assert torch.equal(h, rh) and torch.equal(y, ry)
    assert ops.device_error_flags() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,H,F", [(40, 192, 320), (4, 2560, 1000), (12, 1001, 2560), (20, 2560, 1000)])
def test_ffn_of_any_width_in_smaller_workspaces(M, H, F):
    """The size that AUTO asks for, one byte less, and what the generic kernel needs: the same bits from all."""
    import ctypes as C
    from bitnet_mlx_rs_b200 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(F)
    wg, wu, wd = _weights(g, F, H), _weights(g, F, H), _weights(g, H, F)
    x = torch.randn(M, H, device="cuda", generator=g)
    ry, rh = ops.ffn_forward(wg, 0.05, wu, 0.04, wd, 0.03, x, F, path="generic")
    lib, size = L.load(), {}
    for path in (L.PATH_AUTO, L.PATH_GENERIC):
        n = C.c_size_t()
        assert lib.bitnet_ffn_workspace_size(M, H, F, path, C.byref(n)) == 0
        size[path] = n.value
    ws = torch.empty(max(size.values()) + 256, dtype=torch.uint8, device="cuda")
    base = (ws.data_ptr() + 255) // 256 * 256
    for nbytes in (size[L.PATH_AUTO], size[L.PATH_AUTO] - 1, size[L.PATH_GENERIC]):
        y, h = torch.full_like(x, float("nan")), torch.full((M, F), float("nan"), device="cuda")
        st = lib.bitnet_ffn_forward(wg.data_ptr(), 0.05, wu.data_ptr(), 0.04, wd.data_ptr(), 0.03, x.data_ptr(), h.data_ptr(), y.data_ptr(),
                                    M, H, F, None, base, nbytes, torch.cuda.current_stream().cuda_stream)
        assert st == 0 and torch.equal(h, rh) and torch.equal(y, ry), nbytes
    # the generic kernel's workspace also takes buffers at any address
    xs, ws2 = torch.empty(M * H + 4, device="cuda"), torch.empty(wg.numel() + 16, dtype=torch.uint8, device="cuda")
    xs[1:1 + M * H] = x.view(-1)
    ws2[1:1 + wg.numel()] = wg
    y = torch.full_like(x, float("nan"))
    st = lib.bitnet_ffn_forward(ws2.data_ptr() + 1, 0.05, wu.data_ptr(), 0.04, wd.data_ptr(), 0.03, xs.data_ptr() + 4, h.data_ptr(), y.data_ptr(),
                                M, H, F, None, base, size[L.PATH_GENERIC], torch.cuda.current_stream().cuda_stream)
    assert st == 0 and torch.equal(y, ry)
    assert ops.device_error_flags() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1040, 1088])
def test_odd_width_with_glue_writes_the_activations_anywhere(K):
    import ctypes as C
    from bitnet_mlx_rs_b200 import _lib as L
    M, N = 20, 3000
    g = torch.Generator(device="cuda").manual_seed(K)
    w, x = _weights(g, N, K), torch.randn(M, K, device="cuda", generator=g)
    glue = ops.make_glue(residual=x)
    y, dbg = ops.bitlinear_forward_fused(w, (N,), (0.02,), x, glue=glue, debug=True)
    lib, need = L.load(), C.c_size_t()
    assert lib.bitnet_bitlinear_fused_workspace_size(M, K, N, L.PATH_AUTO, C.byref(need)) == 0
    ws = torch.empty(need.value + 256, dtype=torch.uint8, device="cuda")
    for off in (0, 1, 8):
        q = torch.full((M * K + 16,), 99, dtype=torch.int8, device="cuda")
        opts, y2 = L.ForwardOpts(q_out_dev=q.data_ptr() + off), torch.full_like(y, float("nan"))
        st = lib.bitnet_bitlinear_forward_fused(w.data_ptr(), ops._stack((N,), (0.02,)), x.data_ptr(), C.byref(glue), y2.data_ptr(), M, K,
                                                C.byref(opts), (ws.data_ptr() + 255) // 256 * 256, need.value, torch.cuda.current_stream().cuda_stream)
        assert st == 0 and torch.equal(y2, y)
        assert torch.equal(q[off:off + M * K].view(M, K), dbg["q"]) and bool((q[:off] == 99).all()) and bool((q[off + M * K:] == 99).all())
    assert ops.device_error_flags() == 0
