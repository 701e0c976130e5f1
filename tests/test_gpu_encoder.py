"""GPU parity of the frame encoder: kernels one by one against numpy, and Engine::encode through the C ABI against the
float64 oracle, the golden tokens of the reference's PyTorch oracle and the reference's CPU engine.

Tolerance: fp32 mode max abs error <= 1e-4 on tokens of O(1) magnitude (recipe W5); bf16 / fp16 modes (operands of the
1x1 convolutions rounded to that type, everything else float32) max |err| / max |ref| <= 2e-2."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import dev, load_golden, rel_err, stream_ptr, sync

pytestmark = pytest.mark.gpu

TOL = 1e-4


@pytest.fixture(scope="module")
def L():
    from shield_sisa_b200 import binding
    return binding.load_library(True)


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _hardswish(x):
    return x * np.clip(x + 3.0, 0.0, 6.0) / 6.0


def test_stem_kernel(L):
    import torch
    from oracle import cnn_oracle as CO
    rng = np.random.default_rng(0)
    F = 3
    frames = rng.integers(0, 256, size=(F, 180, 320, 3), dtype=np.uint8)
    frames[0, 0, 0] = (0, 255, 0)                                           # corners exercise the padding taps
    w = (rng.standard_normal((16, 3, 3, 3)) * 0.3).astype(np.float32)
    b = rng.standard_normal(16).astype(np.float32)
    lut = np.stack([((np.arange(256, dtype=np.float32) / np.float32(255)) - CO.MEAN[c]) / CO.STD[c] for c in range(3)])
    w_tap = np.ascontiguousarray(w.transpose(2, 3, 1, 0).reshape(27, 16))   # ((kh*3 + kw)*3 + ci, co)
    out = torch.empty((F, 90, 160, 16), dtype=torch.float32, device="cuda")
    d_frames, d_lut, d_w, d_b = dev(frames), dev(lut.astype(np.float32)), dev(w_tap), dev(b)   # keep the buffers alive
    rc = L.shvk_cnn_stem(_ptr(d_frames), _ptr(d_lut), _ptr(d_w), _ptr(d_b), _ptr(out), F, stream_ptr())
    assert rc == 0
    sync()
    ref = _hardswish(CO.conv_dense(CO.normalise(frames, np.float64), w.astype(np.float64), 3, 2) + b)
    assert np.abs(out.cpu().numpy() - ref).max() < 1e-4


@pytest.mark.parametrize("k,stride,H,W,Cn,act", [(3, 1, 12, 20, 24, 1), (3, 2, 45, 80, 72, 1), (5, 2, 23, 40, 120, 2), (5, 1, 6, 10, 960, 2)])
def test_depthwise_kernel(L, k, stride, H, W, Cn, act):
    import torch
    from oracle import cnn_oracle as CO
    rng = np.random.default_rng(k * 10 + stride)
    F = 2
    x = rng.standard_normal((F, H, W, Cn)).astype(np.float32)
    w = (rng.standard_normal((Cn, 1, k, k)) * 0.4).astype(np.float32)
    b = rng.standard_normal(Cn).astype(np.float32)
    pad = (k - 1) // 2
    Ho, Wo = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    w_tap = np.ascontiguousarray(w.reshape(Cn, k * k).T)
    out = torch.empty((F, Ho, Wo, Cn), dtype=torch.float32, device="cuda")
    d_x, d_w, d_b = dev(x), dev(w_tap), dev(b)
    rc = L.shvk_cnn_depthwise(_ptr(d_x), _ptr(d_w), _ptr(d_b), _ptr(out), F, H, W, Cn, k, stride, Ho, Wo, act, stream_ptr())
    assert rc == 0
    sync()
    ref = CO.conv_depthwise(x.astype(np.float64), w.astype(np.float64), k, stride) + b
    ref = np.maximum(ref, 0) if act == 1 else _hardswish(ref)
    assert np.abs(out.cpu().numpy() - ref).max() < 1e-5
    # wrong output size is refused, not launched
    assert L.shvk_cnn_depthwise(_ptr(d_x), _ptr(d_w), _ptr(d_b), _ptr(out), F, H, W, Cn, k, stride, Ho + 1, Wo, act,
                                stream_ptr()) != 0


@pytest.mark.parametrize("HW,Cn,CS", [(920, 72, 24), (240, 672, 168), (60, 960, 240)])
def test_se_gate_kernel(L, HW, Cn, CS):
    import torch
    rng = np.random.default_rng(HW)
    F = 3
    x = rng.standard_normal((F, HW, Cn)).astype(np.float32)
    w1 = (rng.standard_normal((CS, Cn)) / np.sqrt(Cn)).astype(np.float32)
    b1 = rng.standard_normal(CS).astype(np.float32)
    w2 = (rng.standard_normal((Cn, CS)) / np.sqrt(CS)).astype(np.float32)
    b2 = rng.standard_normal(Cn).astype(np.float32)
    n = L.shvk_cnn_se_partial_floats(F, HW, Cn)
    assert n == F * ((HW + 63) // 64) * Cn
    partial = torch.full((n,), float("nan"), dtype=torch.float32, device="cuda")      # scratch need not be cleared
    gate = torch.empty((F, Cn), dtype=torch.float32, device="cuda")
    args = [dev(x), partial, dev(w1), dev(b1), dev(w2), dev(b2), gate]
    assert L.shvk_cnn_se_gate(*[_ptr(a) for a in args], F, HW, Cn, CS, stream_ptr()) == 0
    sync()
    pooled = x.astype(np.float64).mean(axis=1)
    hid = np.maximum(pooled @ w1.T.astype(np.float64) + b1, 0)
    ref = np.clip(hid @ w2.T.astype(np.float64) + b2 + 3.0, 0, 6) / 6
    got = gate.cpu().numpy()
    assert np.abs(got - ref).max() < 1e-5
    # a frame's gate does not depend on the batch it is in
    gate1 = torch.empty((1, Cn), dtype=torch.float32, device="cuda")
    args1 = [dev(x[1:2]), partial, dev(w1), dev(b1), dev(w2), dev(b2), gate1]
    assert L.shvk_cnn_se_gate(*[_ptr(a) for a in args1], 1, HW, Cn, CS, stream_ptr()) == 0
    sync()
    assert np.array_equal(gate1.cpu().numpy()[0], got[1])


@pytest.mark.parametrize("M,N,K,act,gated,resid", [(14400, 64, 16, 1, False, False), (1000, 24, 72, 0, False, True),
                                                  (120, 160, 960, 0, True, True), (60, 960, 160, 2, False, False),
                                                  (77, 40, 120, 0, True, False)])
def test_pointwise_kernel(L, M, N, K, act, gated, resid):
    import torch
    rng = np.random.default_rng(M + N)
    rows = 60 if gated and M % 60 == 0 else (11 if gated else 1)
    A = rng.standard_normal((M, K)).astype(np.float32)
    Wt = (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32)
    b = rng.standard_normal(N).astype(np.float32)
    gate = rng.uniform(0, 1, size=((M + rows - 1) // rows, K)).astype(np.float32) if gated else None
    R = rng.standard_normal((M, N)).astype(np.float32) if resid else None
    out = dev(R) if resid else torch.empty((M, N), dtype=torch.float32, device="cuda")      # residual in place
    g_dev = dev(gate) if gated else None
    d_a, d_w, d_b = dev(A), dev(Wt), dev(b)
    rc = L.shvk_cnn_pointwise(_ptr(d_a), _ptr(d_w), _ptr(d_b), _ptr(g_dev) if gated else None, rows,
                              _ptr(out) if resid else None, _ptr(out), M, N, K, act, stream_ptr())
    assert rc == 0
    sync()
    a64 = A.astype(np.float64)
    if gated:
        a64 = a64 * np.repeat(gate.astype(np.float64), rows, axis=0)[:M]
    ref = a64 @ Wt.T.astype(np.float64) + b
    ref = np.maximum(ref, 0) if act == 1 else _hardswish(ref) if act == 2 else ref
    if resid:
        ref = ref + R
    assert np.abs(out.cpu().numpy() - ref).max() < 2e-5


@pytest.mark.parametrize("M,N,K,act,gated,resid", [(14400, 64, 16, 1, False, False), (1000, 24, 72, 0, False, True),
                                                  (120, 160, 960, 0, True, True), (60, 960, 160, 2, False, False),
                                                  (77, 40, 120, 0, True, False), (333, 80, 184, 0, False, True),
                                                  (4000, 16, 16, 0, False, True)])
def test_pointwise_tf32_kernel(L, M, N, K, act, gated, resid):
    """Tensor-core form of the 1x1 convolution: operands rounded to TF32 (2^-11 relative), float32 accumulation."""
    import torch
    rng = np.random.default_rng(M + N + 1)
    rows = 60 if gated and M % 60 == 0 else (11 if gated else 1)
    A = rng.standard_normal((M, K)).astype(np.float32)
    Wt = (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32)
    b = rng.standard_normal(N).astype(np.float32)
    gate = rng.uniform(0, 1, size=((M + rows - 1) // rows, K)).astype(np.float32) if gated else None
    R = rng.standard_normal((M, N)).astype(np.float32) if resid else None
    out = dev(R) if resid else torch.empty((M, N), dtype=torch.float32, device="cuda")
    g_dev = dev(gate) if gated else None
    d_a, d_w, d_b = dev(A), dev(Wt), dev(b)
    rc = L.shvk_cnn_pointwise_tf32(_ptr(d_a), _ptr(d_w), _ptr(d_b), _ptr(g_dev) if gated else None, rows,
                                   _ptr(out) if resid else None, _ptr(out), M, N, K, act, stream_ptr())
    assert rc == 0
    sync()
    a64 = A.astype(np.float64)
    if gated:
        a64 = a64 * np.repeat(gate.astype(np.float64), rows, axis=0)[:M]
    ref = a64 @ Wt.T.astype(np.float64) + b
    ref = np.maximum(ref, 0) if act == 1 else _hardswish(ref) if act == 2 else ref
    if resid:
        ref = ref + R
    got = out.cpu().numpy()
    assert np.abs(got - ref).max() < 4e-3                      # |a| |w| sqrt(K) 2^-11 with a ~ N(0,1), w ~ N(0,1/K): about 5e-4
    assert np.abs(got - ref).max() > 0                         # not the exact kernel


@pytest.mark.parametrize("ab,tol", [(1, 2.5e-2), (2, 4e-3)])
@pytest.mark.parametrize("M,N,K,act,gated,resid", [(14400, 64, 16, 1, False, False), (1000, 24, 72, 0, False, True),
                                                  (120, 160, 960, 0, True, True), (60, 960, 160, 2, False, False),
                                                  (77, 40, 120, 0, True, False), (333, 80, 184, 0, False, True),
                                                  (4000, 16, 16, 0, False, True), (700, 384, 960, 0, False, False)])
def test_pointwise_16bit_kernel(L, M, N, K, act, gated, resid, ab, tol):
    """1x1 convolution with operands rounded to bf16 (2^-9 relative) or fp16 (2^-11), float32 accumulation."""
    import torch
    rng = np.random.default_rng(M + N + 2)
    rows = 60 if gated and M % 60 == 0 else (11 if gated else 1)
    A = rng.standard_normal((M, K)).astype(np.float32)
    Wt = (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32)
    b = rng.standard_normal(N).astype(np.float32)
    gate = rng.uniform(0, 1, size=((M + rows - 1) // rows, K)).astype(np.float32) if gated else None
    R = rng.standard_normal((M, N)).astype(np.float32) if resid else None
    out = dev(R) if resid else torch.empty((M, N), dtype=torch.float32, device="cuda")
    g_dev = dev(gate) if gated else None
    d_a, d_w, d_b = dev(A), dev(Wt), dev(b)
    rc = L.shvk_cnn_pointwise_h(_ptr(d_a), _ptr(d_w), _ptr(d_b), _ptr(g_dev) if gated else None, rows,
                                _ptr(out) if resid else None, _ptr(out), M, N, K, act, ab, stream_ptr())
    assert rc == 0
    sync()
    a64 = A.astype(np.float64)
    if gated:
        a64 = a64 * np.repeat(gate.astype(np.float64), rows, axis=0)[:M]
    ref = a64 @ Wt.T.astype(np.float64) + b
    ref = np.maximum(ref, 0) if act == 1 else _hardswish(ref) if act == 2 else ref
    if resid:
        ref = ref + R
    got = out.cpu().numpy()
    assert np.abs(got - ref).max() < tol
    # the same rounding done on the host reproduces the kernel to float32 accumulation error
    dt = torch.bfloat16 if ab == 1 else torch.float16
    a_r = torch.from_numpy(a64.astype(np.float32)).to(dt).double().numpy()
    w_r = torch.from_numpy(Wt).to(dt).double().numpy()
    ref_r = a_r @ w_r.T + b
    ref_r = np.maximum(ref_r, 0) if act == 1 else _hardswish(ref_r) if act == 2 else ref_r
    if resid:
        ref_r = ref_r + R
    assert np.abs(got - ref_r).max() < 5e-5
    assert L.shvk_cnn_pointwise_h(_ptr(d_a), _ptr(d_w), _ptr(d_b), None, 1, None, _ptr(out), M, N, K, act, 0, stream_ptr()) != 0


def test_pool_tokens_kernel(L):
    import torch
    from oracle import cnn_oracle as CO
    rng = np.random.default_rng(5)
    F = 2
    fmap = rng.standard_normal((F, 6, 10, 960)).astype(np.float32)
    out = torch.empty((F, 16, 960), dtype=torch.float32, device="cuda")
    d_map = dev(fmap)
    assert L.shvk_cnn_pool_tokens(_ptr(d_map), _ptr(out), F, stream_ptr()) == 0
    sync()
    ident = {"projection.weight": np.eye(960, dtype=np.float64)}
    ref = CO.tokens_from_map(ident, fmap.astype(np.float64))
    assert np.abs(out.cpu().numpy() - ref).max() < 1e-6


# ---------------------------------------------------------------------------------------------- whole encoder
def _encode(eng, frames, slot=0):
    import torch
    F = frames.shape[0]
    src = dev(frames)
    stream = stream_ptr()
    torch.cuda.synchronize()
    dst = _wrap_u8(eng.frames_ptr(slot), F * 172800)       # device-to-device copy of the crops into the slot buffer
    dst.copy_(src.reshape(-1))
    eng.encode(slot, F, stream)
    sync()
    return _wrap_f32(eng.tokens_ptr(slot), F * 6144).cpu().numpy().reshape(F, 16, 384).copy()


def _wrap(ptr, nbytes, typestr):
    import torch

    class _Arr:
        pass

    a = _Arr()
    a.__cuda_array_interface__ = {"shape": (nbytes // int(typestr[-1]),), "typestr": typestr, "data": (int(ptr), False),
                                  "version": 2}
    return torch.as_tensor(a, device="cuda")


def _wrap_u8(ptr, n):
    return _wrap(ptr, n, "|u1")


def _wrap_f32(ptr, n):
    return _wrap(ptr, n * 4, "<f4")


@pytest.mark.parametrize("case", ["encoder_w5_s3_f11", "encoder_w1_s1_f5"])
@pytest.mark.parametrize("mode", ["fp32", "bf16", "fp16"])
def test_encode_matches_reference(case, mode, weight_files):
    from oracle import cnn_oracle as CO, ref_cpu
    from shield_sisa_b200 import binding, weights as W
    g = load_golden(case)
    path, w = weight_files(str(g["recipe"]), int(g["weight_seed"]))
    frames = W.synth_frames(int(g["frames"]), int(g["frame_seed"]))
    eng = binding.EngineCore(path, mode, max_windows=1, max_frames=4, use_graphs=False)
    tok = _encode(eng, frames)
    assert eng.status() == 0
    # fp32 mode: max abs error <= 1e-4.  16-bit modes (16-bit operands in the 1x1 convolutions): max |err| / max |ref| <= 2e-2
    def err(ref):
        return np.abs(tok - ref).max() if mode == "fp32" else rel_err(tok, ref)
    tol = TOL if mode == "fp32" else 2e-2
    assert err(g["tokens_f64"]) <= tol                                     # reference's PyTorch oracle, float64
    assert err(CO.encode_frames(w, frames, np.float64)) <= tol
    if "tokens_cpu_engine" in g:
        assert err(g["tokens_cpu_engine"]) <= tol                          # reference's CPU engine (stored)
    if ref_cpu.available():
        cpu = ref_cpu.RefCpuEngine(path, threads=2)
        assert err(cpu.encode_frames(frames)) <= tol                       # reference's CPU engine (run here)
        cpu.close()
    print(f"encoder {case} {mode}: err vs float64 oracle {err(g['tokens_f64']):.3e}")
    eng.close()


def test_encode_frame_independence_and_graphs(weight_files):
    """A frame's tokens are bitwise the same alone, in a batch, in another order and through a padded CUDA graph."""
    from shield_sisa_b200 import binding, weights as W
    path, _ = weight_files("W5", 3)
    frames = W.synth_frames(7, 21)
    eager = binding.EngineCore(path, "fp32", max_windows=1, max_frames=16, use_graphs=False)
    graph = binding.EngineCore(path, "fp32", max_windows=1, max_frames=16, use_graphs=True)
    full = _encode(eager, frames)
    assert np.array_equal(_encode(eager, frames[3:4])[0], full[3])
    perm = np.array([6, 2, 0, 5, 1, 4, 3])
    assert np.array_equal(_encode(eager, frames[perm], slot=1), full[perm])
    assert graph.frame_bucket(7) == 8
    assert np.array_equal(_encode(graph, frames), full)
    assert np.array_equal(_encode(graph, frames), full)                    # second launch of the captured graph
    from oracle.cnn_oracle import BLOCKS
    assert eager.encode_launches() == 4 + sum(2 + (1 if e != i else 0) + (2 if se else 0) for (i, _k, e, _o, se, _a, _s) in BLOCKS)
    eager.close()
    graph.close()


@pytest.mark.parametrize("N,K,gated", [(16, 16, False), (24, 64, False), (24, 72, True), (40, 120, True), (72, 24, False), (80, 184, False),
                                       (80, 200, True), (64, 16, False), (112, 480, True), (160, 264, True), (384, 960, False), (672, 112, False)])
def test_pointwise_tiles_give_the_same_rows(L, N, K, gated):
    """The fp32 1x1 convolution picks its tile from the row count (one tile a row, 64 or 128 columns, slabs of 8, 16 or 32 channels
    whose last one may be short): rows are the same bits whatever the tile, and near float64 (K products in float32: the error of
    a sum is below (K + 4) 2^-24 times the sum of magnitudes, first order)."""
    import torch
    rng = np.random.default_rng(N * K)
    big, rows_per_gate = 13001, 240
    a = rng.standard_normal((big, K)).astype(np.float32)
    w, b = (rng.standard_normal((N, K)) / 8).astype(np.float32), rng.standard_normal(N).astype(np.float32)
    g = rng.random(((big + rows_per_gate - 1) // rows_per_gate, K)).astype(np.float32)
    r = rng.standard_normal((big, N)).astype(np.float32)
    A, Wt, Bt, G, R = (torch.from_numpy(x).cuda() for x in (a, w, b, g, r))
    outs = []
    for m in (big, 3333, 65, 1):
        out = torch.full((big, N), 9.0, device="cuda")
        rc = L.shvk_cnn_pointwise(A.data_ptr(), Wt.data_ptr(), Bt.data_ptr(), G.data_ptr() if gated else None, rows_per_gate, R.data_ptr(),
                                  out.data_ptr(), m, N, K, 0, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
        assert (out[m:] == 9.0).all()
        outs.append(out[:m])
    for o in outs[1:]:
        assert torch.equal(o, outs[0][:len(o)])
    rows = np.r_[0:200, big - 200:big]
    x = a[rows].astype(np.float64) * (g[rows // rows_per_gate].astype(np.float64) if gated else 1.0)
    want = x @ w.T.astype(np.float64) + b + r[rows]
    bound = (K + 4) * 2.0 ** -24 * (np.abs(x) @ np.abs(w.T).astype(np.float64) + np.abs(b) + np.abs(r[rows]))
    assert (np.abs(outs[0][torch.from_numpy(rows).cuda()].cpu().numpy() - want) <= bound).all()


# ---------------------------------------------------------------------------------------------- fused kernels (16-bit modes)
def _pack(L, w, order, dtype, n_pad=None, k_pad=None):
    import torch
    n, k = w.shape
    full = np.zeros((n_pad or n, k_pad or k), np.float32)
    full[:n, :k] = w
    out = np.zeros(L.shvk_cnn_packed_bytes(*full.shape, order), np.uint8)
    assert L.shvk_cnn_pack_weights(full.ctypes.data, *full.shape, order, dtype, out.ctypes.data) == 0
    return torch.from_numpy(out).cuda()


_BLOCKS = [(16, 3, 16, 16, False, 1), (16, 3, 64, 24, False, 2), (24, 3, 72, 24, False, 1), (24, 5, 72, 40, True, 2),
           (40, 5, 120, 40, True, 1), (40, 5, 120, 40, True, 1), (40, 3, 240, 80, False, 2), (80, 3, 200, 80, False, 1),
           (80, 3, 184, 80, False, 1), (80, 3, 184, 80, False, 1), (80, 3, 480, 112, True, 1), (112, 3, 672, 112, True, 1),
           (112, 5, 672, 160, True, 2), (160, 5, 960, 160, True, 1), (160, 5, 960, 160, True, 1)]


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("N,K", [(40, 72), (40, 120), (112, 480), (112, 672), (160, 672), (160, 960), (384, 960)])
def test_row_kernels_split_by_channels_give_the_same_rows(L, N, K, dtype):
    """The gated projection and (N = 384) the token projection split few rows by output channels and load ahead: the same bits as
    the unsplit form of many rows, nothing written past the rows."""
    import torch
    rng = np.random.default_rng(N + K)
    tdt = torch.bfloat16 if dtype == 1 else torch.float16
    st = torch.cuda.current_stream().cuda_stream
    big = 64 * 161 + 5
    w = (rng.standard_normal((N, K)) / 16).astype(np.float32)
    a = rng.standard_normal((big, K)).astype(np.float32)
    outs = []
    if N == 384:
        A, P = torch.from_numpy(a).cuda().to(tdt), _pack(L, w, 2, dtype)
    else:
        A, P = torch.from_numpy(a).cuda(), _pack(L, w, 1, dtype, k_pad=(K + 15) // 16 * 16)
        G = torch.rand((big + 59) // 60, K, device="cuda")
        R, b = torch.randn(big, N, device="cuda"), torch.randn(N, device="cuda")
    for m in (big, 5000, 77, 1):
        out = torch.full((big, N), 9.0, device="cuda")
        if N == 384:
            assert L.shvk_cnn_token_proj(A.data_ptr(), P.data_ptr(), out.data_ptr(), m, dtype, st) == 0
        else:
            assert L.shvk_cnn_rows_gate(A.data_ptr(), P.data_ptr(), b.data_ptr(), G.data_ptr(), 60, R.data_ptr(), out.data_ptr(), m, N, K, dtype, st) == 0
        torch.cuda.synchronize()
        assert (out[m:] == 9.0).all()
        outs.append(out[:m])
    for o in outs[1:]:
        assert torch.equal(o, outs[0][:len(o)])


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("N,K", [(40, 120), (112, 100), (112, 672), (160, 36), (160, 960)])
def test_row_kernel_tiles_give_the_same_rows(L, N, K, dtype):
    """The gated projection of many rows reads through a ring of shared memory, in blocks of four to eight warps by the row count: the
    bits of the form for few rows, with an odd number of k tiles and a ragged last one, frames of 60 rows and of 7, with and
    without a residual, nothing written past the rows."""
    import torch
    st = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(N * K)
    big, part = 148 * 128 + 64 * 148 + 5, 9000                 # `part` rows are few
    P = _pack(L, (rng.standard_normal((N, K)) / 16).astype(np.float32), 1, dtype, k_pad=(K + 15) // 16 * 16)
    A, R, b = torch.randn(big, K, device="cuda"), torch.randn(big, N, device="cuda"), torch.randn(N, device="cuda")
    for gate_rows, res in ((60, True), (7, False)):
        G = torch.rand((big + gate_rows - 1) // gate_rows, K, device="cuda")
        call = lambda a, g, r, out, m: L.shvk_cnn_rows_gate(a.data_ptr(), P.data_ptr(), b.data_ptr(), g.data_ptr(), gate_rows,  # noqa: E731
                                                            r.data_ptr() if res else None, out.data_ptr(), m, N, K, dtype, st)
        want = torch.empty(big, N, device="cuda")
        step = part // (gate_rows * 4) * gate_rows * 4          # whole frames, 16-byte aligned
        for m0 in range(0, big, step):
            assert call(A[m0:], G[m0 // gate_rows:], R[m0:], want[m0:], min(step, big - m0)) == 0
        for m in (big, 148 * 112, 148 * 96 + 1, 148 * 80 - 3, 148 * 144, 10321):
            out = torch.full((big, N), 9.0, device="cuda")
            assert call(A, G, R, out, m) == 0
            torch.cuda.synchronize()
            assert torch.equal(out[:m], want[:m]) and (out[m:] == 9.0).all()


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("block", [2, 3, 4, 5, 7, 8, 9, 11, 12, 13, 14])
def test_fused_block_matches_layers(L, block, dtype):
    """One fused block (expand + depthwise + project or pooled sums, gate, gated project) against the layer kernels on the same
    input, within what operands that round the other way would cost: an ulp of the 16-bit type (at most 2^-7 or 2^-10 relative) on
    isolated terms of a K-term sum.  (That they do not, bit for bit, is tested further down.)"""
    import torch
    cin, k, cexp, cout, se, stride = _BLOCKS[block - 1]
    H, W = 90, 160
    for _cin, kk, *_r, st in _BLOCKS[:block - 1]:
        H, W = (H + 2 * ((kk - 1) // 2) - kk) // st + 1, (W + 2 * ((kk - 1) // 2) - kk) // st + 1
    pad = (k - 1) // 2
    Ho, Wo = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    act = 1 if block < 7 else 2
    rng = np.random.default_rng(block)
    F = 3
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)  # noqa: E731
    x, we, be = dev(f32(F, H, W, cin)), f32(cexp, cin) / np.float32(np.sqrt(cin)), dev(f32(cexp))
    wd, bd = dev(f32(k * k, cexp) / np.float32(k)), dev(f32(cexp))
    wp, bp = f32(cout, cexp) / np.float32(np.sqrt(cexp)), dev(f32(cout))
    zeros = lambda *s: torch.zeros(s, device="cuda")  # noqa: E731
    # layer by layer
    E, Dm, Y = zeros(F, H, W, cexp), zeros(F, Ho, Wo, cexp), zeros(F, Ho, Wo, cout)
    d_we, d_wp = dev(we), dev(wp)
    assert L.shvk_cnn_pointwise_h(_ptr(x), _ptr(d_we), _ptr(be), None, 1, None, _ptr(E), F * H * W, cexp, cin, act, dtype, stream_ptr()) == 0
    assert L.shvk_cnn_depthwise(_ptr(E), _ptr(wd), _ptr(bd), _ptr(Dm), F, H, W, cexp, k, stride, Ho, Wo, act, stream_ptr()) == 0
    res = x if stride == 1 and cin == cout else None
    gate = zeros(F, cexp)
    if se:
        cs = {72: 24, 120: 32, 480: 120, 672: 168, 960: 240}[cexp]
        w1, b1, w2, b2 = dev(f32(cs, cexp) / np.float32(np.sqrt(cexp))), dev(f32(cs)), dev(f32(cexp, cs) / np.float32(np.sqrt(cs))), dev(f32(cexp))
        part = zeros(L.shvk_cnn_se_partial_floats(F, Ho * Wo, cexp))
        assert L.shvk_cnn_se_gate(_ptr(Dm), _ptr(part), _ptr(w1), _ptr(b1), _ptr(w2), _ptr(b2), _ptr(gate), F, Ho * Wo, cexp, cs, stream_ptr()) == 0
    assert L.shvk_cnn_pointwise_h(_ptr(Dm), _ptr(d_wp), _ptr(bp), _ptr(gate) if se else None, Ho * Wo, _ptr(res) if res is not None else None,
                                  _ptr(Y), F * Ho * Wo, cout, cexp, 0, dtype, stream_ptr()) == 0
    # fused
    cols, kp = C.c_int(), C.c_int()
    L.shvk_cnn_block_padding(block, C.byref(cols), C.byref(kp))
    tiles = L.shvk_cnn_block_tiles(block)
    assert (tiles > 0) == se and cols.value >= cexp and kp.value >= cexp
    p_we = _pack(L, we, 0, dtype, cols.value)
    p_wp = _pack(L, wp, 1 if se else 0, dtype, None, kp.value)
    out = zeros(F, Ho, Wo, cexp if se else cout)
    sums = torch.full((F, max(tiles, 1), cexp), float("nan"), device="cuda")
    args = [block, _ptr(x), _ptr(p_we), _ptr(be), _ptr(wd), _ptr(bd), None if se else _ptr(p_wp), None if se else _ptr(bp)]
    assert L.shvk_cnn_block(*args, _ptr(out), _ptr(sums), F, dtype, stream_ptr()) == 0
    assert L.shvk_cnn_block(*args, _ptr(x), _ptr(sums), F, dtype, stream_ptr()) != 0        # in place is refused
    if se:
        sync()
        assert rel_err(out.cpu().numpy(), Dm.cpu().numpy()) < 2e-6                            # float32 arithmetic on the same mma sums
        assert rel_err(sums.sum(1).cpu().numpy(), Dm.sum((1, 2)).cpu().numpy()) < 1e-5
        g2, y2 = zeros(F, cexp), zeros(F, Ho, Wo, cout)
        assert L.shvk_cnn_se_gate_sums(_ptr(sums), _ptr(w1), _ptr(b1), _ptr(w2), _ptr(b2), _ptr(g2), F, tiles, Ho * Wo, cexp, cs, stream_ptr()) == 0
        assert L.shvk_cnn_rows_gate(_ptr(out), _ptr(p_wp), _ptr(bp), _ptr(g2), Ho * Wo, _ptr(res) if res is not None else None, _ptr(y2),
                                    F * Ho * Wo, cout, cexp, dtype, stream_ptr()) == 0
        sync()
        assert np.abs((g2 - gate).cpu().numpy()).max() < 1e-5
        out = y2
    sync()
    got, ref = out.cpu().numpy(), Y.cpu().numpy()
    unit = 2.0 ** -8 if dtype == 1 else 2.0 ** -11
    assert np.abs(got - ref).max() < 4 * unit * float(Dm.abs().max()) * np.abs(wp).max()   # two operands rounded the other way, an ulp each
    assert np.sqrt(((got - ref) ** 2).mean() / (ref ** 2).mean()) < unit / 16
    # a frame's result does not depend on the batch it is in
    one, s1 = zeros(1, *[int(v) for v in (Ho, Wo, cexp if se else cout)]), zeros(1, max(tiles, 1), cexp)
    x1 = x[2:3].contiguous()
    assert L.shvk_cnn_block(block, _ptr(x1), *args[2:], _ptr(one), _ptr(s1), 1, dtype, stream_ptr()) == 0
    sync()
    if se:
        assert torch.equal(s1[0], sums[2])
    else:
        assert torch.equal(one[0], out[2])


@pytest.mark.parametrize("dtype", [1, 2])
def test_fused_ends_of_the_encoder(L, dtype):
    """Stem + block 1 and last convolution + pooling + token projection against the layer kernels."""
    import torch
    from oracle import cnn_oracle as CO
    rng = np.random.default_rng(9)
    F = 3
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)  # noqa: E731
    zeros = lambda *s: torch.zeros(s, device="cuda")  # noqa: E731
    unit = 2.0 ** -8 if dtype == 1 else 2.0 ** -11
    frames = dev(rng.integers(0, 256, size=(F, 180, 320, 3), dtype=np.uint8))
    lut = np.stack([((np.arange(256, dtype=np.float32) / np.float32(255)) - CO.MEAN[c]) / CO.STD[c] for c in range(3)]).astype(np.float32)
    ws, bs, wd, bd, wp, bp = f32(27, 16) * np.float32(0.3), f32(16), dev(f32(9, 16) / 3), dev(f32(16)), f32(16, 16) / 4, dev(f32(16))
    d_lut, d_ws, d_bs, d_wp = dev(lut), dev(ws), dev(bs), dev(wp)
    S, Dm, Y, out = zeros(F, 90, 160, 16), zeros(F, 90, 160, 16), zeros(F, 90, 160, 16), zeros(F, 90, 160, 16)
    assert L.shvk_cnn_stem(_ptr(frames), _ptr(d_lut), _ptr(d_ws), _ptr(d_bs), _ptr(S), F, stream_ptr()) == 0
    assert L.shvk_cnn_depthwise(_ptr(S), _ptr(wd), _ptr(bd), _ptr(Dm), F, 90, 160, 16, 3, 1, 90, 160, 1, stream_ptr()) == 0
    assert L.shvk_cnn_pointwise_h(_ptr(Dm), _ptr(d_wp), _ptr(bp), None, 1, _ptr(S), _ptr(Y), F * 14400, 16, 16, 0, dtype, stream_ptr()) == 0
    p_wp = _pack(L, wp, 0, dtype)
    assert L.shvk_cnn_stem_block(_ptr(frames), _ptr(d_lut), ws.ctypes.data, bs.ctypes.data, _ptr(wd), _ptr(bd), _ptr(p_wp), _ptr(bp),
                                 _ptr(out), F, dtype, stream_ptr()) == 0
    sync()
    assert float((out - Y).abs().max()) < 2 * unit * float(Dm.abs().max()) * np.abs(wp).max()   # one operand rounded the other way: one ulp
    assert float(((out - Y) ** 2).mean().sqrt() / (Y ** 2).mean().sqrt()) < unit / 64
    x, wl, bl, wt = dev(f32(F, 60, 160)), f32(960, 160) / np.float32(np.sqrt(160)), dev(f32(960)), f32(384, 960) / np.float32(np.sqrt(960))
    fmap, pooled, tok = zeros(F, 60, 960), zeros(F, 16, 960), zeros(F * 16, 384)
    d_wl, d_wt = dev(wl), dev(wt)
    assert L.shvk_cnn_pointwise_h(_ptr(x), _ptr(d_wl), _ptr(bl), None, 1, None, _ptr(fmap), F * 60, 960, 160, 2, dtype, stream_ptr()) == 0
    assert L.shvk_cnn_pool_tokens(_ptr(fmap), _ptr(pooled), F, stream_ptr()) == 0
    assert L.shvk_cnn_pointwise_h(_ptr(pooled), _ptr(d_wt), None, None, 1, None, _ptr(tok), F * 16, 384, 960, 0, dtype, stream_ptr()) == 0
    p_wl, p_wt = _pack(L, wl, 0, dtype), _pack(L, wt, 2, dtype)
    low = torch.zeros((F, 16, 960), device="cuda", dtype=torch.bfloat16 if dtype == 1 else torch.float16)
    tok2 = zeros(F * 16, 384)
    assert L.shvk_cnn_last_pool(_ptr(x), _ptr(p_wl), _ptr(bl), _ptr(low), F, dtype, stream_ptr()) == 0
    assert L.shvk_cnn_token_proj(_ptr(low), _ptr(p_wt), _ptr(tok2), F * 16, dtype, stream_ptr()) == 0
    sync()
    assert rel_err(low.float().cpu().numpy(), pooled.cpu().numpy()) < unit
    assert rel_err(tok2.cpu().numpy(), tok.cpu().numpy()) < unit


def _block_both_ways(L, block, dtype, F, seed=0):
    """Block `block` of the network on F frames of random maps, by the layer kernels and by the fused ones.  Returns (layers, fused),
    each a dict of out (the block's map, or behind a gate the depthwise map) and, where the block has a gate, sums, gate and y (the
    gated projection)."""
    import torch
    cin, k, cexp, cout, se, stride = _BLOCKS[block - 1]
    H, W = 90, 160
    for _cin, kk, *_r, st in _BLOCKS[:block - 1]:
        H, W = (H + 2 * ((kk - 1) // 2) - kk) // st + 1, (W + 2 * ((kk - 1) // 2) - kk) // st + 1
    pad = (k - 1) // 2
    Ho, Wo = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    act = 1 if block < 7 else 2
    gen = torch.Generator(device="cuda").manual_seed(100 * block + seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    zeros = lambda *s: torch.zeros(s, device="cuda")  # noqa: E731
    x, we, be = 2 * rn(F, H, W, cin), rn(cexp, cin) / cin ** 0.5, rn(cexp)
    wd, bd, wp, bp = rn(k * k, cexp) / k, rn(cexp), rn(cout, cexp) / cexp ** 0.5, rn(cout)
    res = x if stride == 1 and cin == cout else None
    E, a, f = zeros(F, H, W, cexp), {}, {}
    dw = zeros(F, Ho, Wo, cexp)
    assert L.shvk_cnn_pointwise_h(_ptr(x), _ptr(we), _ptr(be), None, 1, None, _ptr(E), F * H * W, cexp, cin, act, dtype, stream_ptr()) == 0
    assert L.shvk_cnn_depthwise(_ptr(E), _ptr(wd), _ptr(bd), _ptr(dw), F, H, W, cexp, k, stride, Ho, Wo, act, stream_ptr()) == 0
    if se:
        cs = {72: 24, 120: 32, 480: 120, 672: 168, 960: 240}[cexp]
        w1, b1, w2, b2 = rn(cs, cexp) / cexp ** 0.5, rn(cs), rn(cexp, cs) / cs ** 0.5, rn(cexp)
        a["sums"] = zeros(F, L.shvk_cnn_se_partial_floats(1, Ho * Wo, cexp) // cexp, cexp)
        a["gate"] = zeros(F, cexp)
        assert L.shvk_cnn_se_gate(_ptr(dw), _ptr(a["sums"]), _ptr(w1), _ptr(b1), _ptr(w2), _ptr(b2), _ptr(a["gate"]), F, Ho * Wo, cexp, cs,
                                  stream_ptr()) == 0
    y = zeros(F, Ho, Wo, cout)
    assert L.shvk_cnn_pointwise_h(_ptr(dw), _ptr(wp), _ptr(bp), _ptr(a["gate"]) if se else None, Ho * Wo, _ptr(res) if res is not None else None,
                                  _ptr(y), F * Ho * Wo, cout, cexp, 0, dtype, stream_ptr()) == 0
    a["out"] = dw if se else y
    cols, kp = C.c_int(), C.c_int()
    L.shvk_cnn_block_padding(block, C.byref(cols), C.byref(kp))
    p_we, p_wp = _pack(L, we.cpu().numpy(), 0, dtype, cols.value), _pack(L, wp.cpu().numpy(), 1 if se else 0, dtype, None, kp.value)
    tiles = L.shvk_cnn_block_tiles(block)
    f["out"], f["sums"] = zeros(F, Ho, Wo, cexp if se else cout), torch.full((F, max(tiles, 1), cexp), float("nan"), device="cuda")
    assert L.shvk_cnn_block(block, _ptr(x), _ptr(p_we), _ptr(be), _ptr(wd), _ptr(bd), None if se else _ptr(p_wp), None if se else _ptr(bp),
                            _ptr(f["out"]), _ptr(f["sums"]), F, dtype, stream_ptr()) == 0
    if se:
        a["y"], f["y"], f["gate"] = y, zeros(F, Ho, Wo, cout), zeros(F, cexp)
        assert L.shvk_cnn_se_gate_sums(_ptr(f["sums"]), _ptr(w1), _ptr(b1), _ptr(w2), _ptr(b2), _ptr(f["gate"]), F, tiles, Ho * Wo, cexp, cs,
                                       stream_ptr()) == 0
        assert L.shvk_cnn_rows_gate(_ptr(f["out"]), _ptr(p_wp), _ptr(bp), _ptr(f["gate"]), Ho * Wo, _ptr(res) if res is not None else None,
                                    _ptr(f["y"]), F * Ho * Wo, cout, cexp, dtype, stream_ptr()) == 0
    sync()
    return a, f


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("block", [2, 3, 4, 5, 7, 8, 9, 11, 12, 13, 14])
def test_fused_block_gives_the_bits_of_the_layers(L, block, dtype):
    """Expand, depthwise and (no gate between) projection in one kernel: every step rounds as the layer kernels round it, so the maps
    are the same bits."""
    import torch
    a, f = _block_both_ways(L, block, dtype, 3)
    assert torch.equal(f["out"], a["out"])


@pytest.mark.parametrize("block,frames", [(7, (37, 38)), (8, (18, 19, 74, 75)), (9, (18, 19, 74, 75))])
def test_whole_block_gives_the_bits_of_the_layers_on_every_tile(L, block, frames):
    """The deeper whole blocks take smaller tiles of a map for few frames: both sides of the lines (on 148 SMs)."""
    import torch
    for F in frames:
        for dtype in (1, 2):
            a, f = _block_both_ways(L, block, dtype, F, seed=F)
            assert torch.equal(f["out"], a["out"]), (F, dtype)


@pytest.mark.parametrize("dtype", [1, 2])
def test_fused_ends_give_the_bits_of_the_layers(L, dtype):
    """Stem + block 1, and last convolution + pooling (rounded to the 16-bit type, as the token projection rounds its operand)."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(5)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    zeros = lambda *s: torch.zeros(s, device="cuda")  # noqa: E731
    F, tdt = 3, torch.bfloat16 if dtype == 1 else torch.float16
    frames = torch.randint(0, 256, (F, 180, 320, 3), device="cuda", generator=gen, dtype=torch.uint8)
    lut, ws, bs, wd, bd, wp, bp = 1.3 * rn(3, 256), 0.3 * rn(27, 16), rn(16), rn(9, 16) / 3, rn(16), rn(16, 16) / 4, rn(16)
    s, dw, y, out = zeros(F, 90, 160, 16), zeros(F, 90, 160, 16), zeros(F, 90, 160, 16), zeros(F, 90, 160, 16)
    assert L.shvk_cnn_stem(_ptr(frames), _ptr(lut), _ptr(ws), _ptr(bs), _ptr(s), F, stream_ptr()) == 0
    assert L.shvk_cnn_depthwise(_ptr(s), _ptr(wd), _ptr(bd), _ptr(dw), F, 90, 160, 16, 3, 1, 90, 160, 1, stream_ptr()) == 0
    assert L.shvk_cnn_pointwise_h(_ptr(dw), _ptr(wp), _ptr(bp), None, 1, _ptr(s), _ptr(y), F * 14400, 16, 16, 0, dtype, stream_ptr()) == 0
    p_wp, h_ws, h_bs = _pack(L, wp.cpu().numpy(), 0, dtype), ws.cpu().numpy(), bs.cpu().numpy()
    assert L.shvk_cnn_stem_block(_ptr(frames), _ptr(lut), h_ws.ctypes.data, h_bs.ctypes.data, _ptr(wd), _ptr(bd), _ptr(p_wp), _ptr(bp),
                                 _ptr(out), F, dtype, stream_ptr()) == 0
    sync()
    assert torch.equal(out, y)
    x, wl, bl = 2 * rn(F, 60, 160), rn(960, 160) / 160 ** 0.5, rn(960)
    fmap, pooled, low = zeros(F, 60, 960), zeros(F, 16, 960), torch.zeros((F, 16, 960), device="cuda", dtype=tdt)
    assert L.shvk_cnn_pointwise_h(_ptr(x), _ptr(wl), _ptr(bl), None, 1, None, _ptr(fmap), F * 60, 960, 160, 2, dtype, stream_ptr()) == 0
    assert L.shvk_cnn_pool_tokens(_ptr(fmap), _ptr(pooled), F, stream_ptr()) == 0
    p_wl = _pack(L, wl.cpu().numpy(), 0, dtype)
    assert L.shvk_cnn_last_pool(_ptr(x), _ptr(p_wl), _ptr(bl), _ptr(low), F, dtype, stream_ptr()) == 0
    sync()
    assert torch.equal(low, pooled.to(tdt))


def test_stem_block_takes_crops_at_any_address(L):
    """Crops are read in words where their address allows, in bytes where it does not: the same map."""
    import torch
    frames = torch.randint(0, 256, (2, 180, 320, 3), device="cuda", dtype=torch.uint8)
    lut, wd, bd, bp = (torch.randn(*n, device="cuda") for n in ((3, 256), (9, 16), (16,), (16,)))
    ws, bs = np.random.default_rng(1).standard_normal((27, 16)).astype(np.float32), np.zeros(16, np.float32)
    p_wp = _pack(L, np.random.default_rng(2).standard_normal((16, 16)).astype(np.float32), 0, 1)
    outs = []
    for shift in range(4):
        moved = torch.zeros(frames.numel() + 4, device="cuda", dtype=torch.uint8)
        moved[shift:shift + frames.numel()] = frames.reshape(-1)
        out = torch.empty(2, 90, 160, 16, device="cuda")
        assert L.shvk_cnn_stem_block(moved.data_ptr() + shift, _ptr(lut), ws.ctypes.data, bs.ctypes.data, _ptr(wd), _ptr(bd), _ptr(p_wp), _ptr(bp),
                                     _ptr(out), 2, 1, stream_ptr()) == 0
        sync()
        outs.append(out)
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("rows", [16, 80, 77, 5136])
def test_token_projection_gives_the_bits_of_the_layer(L, rows, dtype):
    """The token projection sums 16 values of k to an mma in ascending order, in both its forms (rows up to 5,120 split by channels), as the
    16-bit 1x1 layer does."""
    import torch
    tdt = torch.bfloat16 if dtype == 1 else torch.float16
    gen = torch.Generator(device="cuda").manual_seed(rows)
    a, w = (torch.randn(n, 960, device="cuda", generator=gen) for n in (rows, 384))
    low, got, want = a.to(tdt), torch.zeros(rows, 384, device="cuda"), torch.zeros(rows, 384, device="cuda")
    p_w = _pack(L, w.cpu().numpy(), 2, dtype)
    assert L.shvk_cnn_token_proj(_ptr(low), _ptr(p_w), _ptr(got), rows, dtype, stream_ptr()) == 0
    assert L.shvk_cnn_pointwise_h(_ptr(a), _ptr(w), None, None, 1, None, _ptr(want), rows, 384, 960, 0, dtype, stream_ptr()) == 0
    sync()
    assert torch.equal(got, want)


@pytest.mark.parametrize("Cn,CS", [(72, 24), (120, 32), (480, 120), (672, 168), (960, 240), (64, 18)])
def test_se_gate_forms_give_the_same_bits(L, Cn, CS):
    """A gate comes from a cluster of blocks while four frames fit its shared memory (below 3,072 channels in both layers), else from one block.
    Channels of zeros take the same layer to the second form: the same bits.  Frame counts: one and four frames a cluster, the last
    one partly filled, one and four outputs of a warp at a time."""
    import torch
    HW, wide, Fmax = 60, 3072, 151
    gen = torch.Generator(device="cuda").manual_seed(Cn)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    x, w1, b1, w2, b2 = rn(Fmax, HW, Cn), rn(CS, Cn) / Cn ** 0.5, rn(CS), rn(Cn, CS) / CS ** 0.5, rn(Cn)

    def pad(t, *shape):
        out = torch.zeros(shape, device="cuda")
        out[tuple(slice(0, n) for n in t.shape)] = t
        return out

    big = (pad(x, Fmax, HW, wide), pad(w1, CS, wide), b1, pad(w2, wide, CS), pad(b2, wide))

    def gate(args, F, ch):
        x_, w1_, b1_, w2_, b2_ = args
        part, out = torch.zeros(L.shvk_cnn_se_partial_floats(F, HW, ch), device="cuda"), torch.full((Fmax, ch), 9.0, device="cuda")
        assert L.shvk_cnn_se_gate(_ptr(x_), _ptr(part), _ptr(w1_), _ptr(b1_), _ptr(w2_), _ptr(b2_), _ptr(out), F, HW, ch, CS, stream_ptr()) == 0
        sync()
        assert (out[F:] == 9.0).all()
        return out[:F, :Cn]

    want = gate(big, Fmax, wide)
    for F in (1, 3, 55, 57, 75, 148, Fmax):
        assert torch.equal(gate((x, w1, b1, w2, b2), F, Cn), want[:F])


@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("block", [4, 5, 11, 12, 13, 14])
def test_gated_block_gives_the_bits_of_the_layers(L, block, dtype):
    """Behind a gate: the pooled sums (groups of 64 pixels, eight partial sums each), the gate and the gated projection are the bits of the
    layer kernels, whatever share of the channels a thread block walks: one chunk (3 frames), several (38 to 150 frames, by block) or
    all of them (600 frames); the gate's forms change in the same range."""
    import torch
    for F in (3, 38, 75, 150, 600):
        a, f = _block_both_ways(L, block, dtype, F, seed=F)
        for name in ("out", "sums", "gate", "y"):
            assert torch.equal(f[name], a[name]), (F, name)


@pytest.mark.parametrize("block", [2, 3, 7, 8, 9])
def test_fused_block_keeps_infinities(L, block):
    """A pixel beyond fp16's range rounds to infinity as an operand: with positive weights every output it reaches is infinite, in the
    layers and in the fused block alike; the channels that only pad the last chunk (blocks 8 to 10) must not make it NaN."""
    import torch
    cin, k, cexp, cout, _se, stride = _BLOCKS[block - 1]
    H, W = 90, 160
    for _cin, kk, *_r, st in _BLOCKS[:block - 1]:
        H, W = (H + 2 * ((kk - 1) // 2) - kk) // st + 1, (W + 2 * ((kk - 1) // 2) - kk) // st + 1
    pad = (k - 1) // 2
    Ho, Wo = (H + 2 * pad - k) // stride + 1, (W + 2 * pad - k) // stride + 1
    act = 1 if block < 7 else 2
    gen = torch.Generator(device="cuda").manual_seed(block)
    rp = lambda *s: torch.rand(*s, device="cuda", generator=gen) * 0.05 + 0.01  # noqa: E731
    zeros = lambda *s: torch.zeros(s, device="cuda")  # noqa: E731
    x, we, be, wd, bd, wp, bp = rp(1, H, W, cin), rp(cexp, cin), rp(cexp), rp(k * k, cexp), rp(cexp), rp(cout, cexp), rp(cout)
    x[0, 5, 7] = 1e5
    res = x if stride == 1 and cin == cout else None
    E, dw, y, out = zeros(1, H, W, cexp), zeros(1, Ho, Wo, cexp), zeros(1, Ho, Wo, cout), zeros(1, Ho, Wo, cout)
    assert L.shvk_cnn_pointwise_h(_ptr(x), _ptr(we), _ptr(be), None, 1, None, _ptr(E), H * W, cexp, cin, act, 2, stream_ptr()) == 0
    assert L.shvk_cnn_depthwise(_ptr(E), _ptr(wd), _ptr(bd), _ptr(dw), 1, H, W, cexp, k, stride, Ho, Wo, act, stream_ptr()) == 0
    assert L.shvk_cnn_pointwise_h(_ptr(dw), _ptr(wp), _ptr(bp), None, 1, _ptr(res) if res is not None else None, _ptr(y), Ho * Wo, cout, cexp, 0,
                                  2, stream_ptr()) == 0
    cols, kp = C.c_int(), C.c_int()
    L.shvk_cnn_block_padding(block, C.byref(cols), C.byref(kp))
    p_we, p_wp = _pack(L, we.cpu().numpy(), 0, 2, cols.value), _pack(L, wp.cpu().numpy(), 0, 2, None, kp.value)
    assert L.shvk_cnn_block(block, _ptr(x), _ptr(p_we), _ptr(be), _ptr(wd), _ptr(bd), _ptr(p_wp), _ptr(bp), _ptr(out), None, 1, 2, stream_ptr()) == 0
    sync()
    assert torch.isinf(y).any() and not torch.isnan(y).any()
    assert torch.equal(out, y)


@pytest.mark.parametrize("mode", ["bf16", "fp16"])
def test_fused_encode_frame_independence_and_graphs(mode, weight_files):
    """16-bit modes: a frame's tokens are bitwise the same alone, in batches of every size at which a fused kernel changes its form
    (shares of channels, frames to a cluster, split row kernels), in another order, and through a padded CUDA graph."""
    from shield_sisa_b200 import binding, weights as W
    path, _ = weight_files("W5", 3)
    frames = W.synth_frames(300, 23)
    eager = binding.EngineCore(path, mode, max_windows=1, max_frames=300, use_graphs=False)
    graph = binding.EngineCore(path, mode, max_windows=1, max_frames=300, use_graphs=True)
    full = _encode(eager, frames)
    assert np.isfinite(full).all()
    for n in (1, 4, 39, 57, 75, 111, 151):
        assert np.array_equal(_encode(eager, frames[:n], slot=n % 2), full[:n])
    for i in (38, 150, 299):
        assert np.array_equal(_encode(eager, frames[i:i + 1])[0], full[i])
    perm = np.random.default_rng(1).permutation(300)
    assert np.array_equal(_encode(eager, frames[perm], slot=1), full[perm])
    for n in (300, 75, 7):
        assert np.array_equal(_encode(graph, frames[:n]), full[:n])
        assert np.array_equal(_encode(graph, frames[perm[:n]]), full[perm[:n]])          # the captured graph on other crops
    eager.close()
    graph.close()
