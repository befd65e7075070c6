"""The engine below the model: op lists of a few GEMVs over hand-made rows."""
import ctypes as C

import numpy as np
import pytest

from amd_c_b200 import synth

pytestmark = pytest.mark.gpu
NONE = (1 << 64) - 1


class Engine:
    """An engine with its own arena and matrices, run on op lists given as (matrix, offset of the Q8 rows, stride, offset of the
    result, stride)."""

    def __init__(self, arena_bytes: int, T: int):
        from amd_c_b200 import _lib

        self.lib, self.T, self.arena = _lib.load(), T, arena_bytes
        self.h, self.keep = C.c_void_p(), []
        d = _lib.EngineDesc(1, 1, 64, T, 1, T, 16, 1e-5, 0, 0, arena_bytes + 64 * T, arena_bytes, arena_bytes, 64, 8)
        self.check(self.lib.ie_b200_engine_create(C.byref(d), C.byref(self.h)))

    def check(self, r):
        from amd_c_b200._lib import check

        check(r)

    def add(self, m) -> int:
        self.keep.append(m)
        return self.lib.ie_b200_engine_add_mat_device(self.h, m.kind, m.rows, m.cols, m.data.data_ptr())

    def write(self, off: int, row: np.ndarray):
        row = np.ascontiguousarray(row)
        self.check(self.lib.ie_b200_engine_write_rows(self.h, off, row.nbytes, 0, 1, row.ctypes.data_as(C.c_void_p)))

    def read(self, off: int, n: int) -> np.ndarray:
        out = np.zeros(n, np.float32)
        self.check(self.lib.ie_b200_engine_read_rows(self.h, off, 4 * n, 0, 1, out.ctypes.data_as(C.c_void_p)))
        return out

    def run(self, gemvs, T=None):
        from amd_c_b200._lib import Op
        from amd_c_b200.backend import OP_GEMV

        ops = [Op(OP_GEMV, m, -1, -1, 0, 0, a, b, NONE, NONE, NONE, a_s, b_s, 0, 0, 0) for m, a, a_s, b, b_s in gemvs]
        self.check(self.lib.ie_b200_engine_set_ops(self.h, (Op * len(ops))(*ops), len(ops), len(ops)))
        T = T or self.T
        toks, out = np.zeros(T, np.uint32), np.zeros(T, np.uint32)
        self.check(self.lib.ie_b200_engine_run(self.h, toks.ctypes.data_as(C.c_void_p), T, 0, 1, out.ctypes.data_as(C.c_void_p), None))

    def close(self):
        self.lib.ie_b200_engine_destroy(self.h)


def _q8(torch, K, rng, T, cols, cuda):
    return K.quant_q8(torch.from_numpy(rng.standard_normal((T, cols)).astype(np.float32)).to(cuda)).cpu().numpy()


def test_expanded_activations_are_shared_only_where_they_still_hold(cuda):
    """GEMMs over the same Q8 rows, one after the other, share the expanded activations: bit for bit what each gives in a run of its
    own. Not where another GEMM's rows come between, and not where the first one's result lies over the Q8 rows, here with token
    rows 256 MB apart, so that the extent of 26 of them (6.7 GB) does not fit 32 bits."""
    import torch

    from amd_c_b200 import kernels as K

    rng = np.random.default_rng(8)
    T, cols, rows, S = 26, 4096, 16, 1 << 28
    e = Engine(26 * S, T)
    mats = [e.add(K.Mat.from_gguf(t, torch.from_numpy(np.ascontiguousarray(synth.make_gguf_bytes(t, rng, rows, cols))).to(cuda), rows, cols))
            for t in (synth.GGML_Q4_K, synth.GGML_Q4_K, synth.GGML_Q6_K)]
    x, z = _q8(torch, K, rng, T, cols, cuda), _q8(torch, K, rng, T, cols, cuda)
    zoff = 1 << 20  # of the other rows, behind the first ones of the same token

    def fill():
        for t in range(T):
            e.write(S * t, x[t]), e.write(S * t + zoff, z[t])

    def results(ops):
        return [np.stack([e.read(b + bs * t, rows) for t in range(T)]).view(np.uint32) for _, _, _, b, bs in ops]

    beside = [(mats[i], 0, S, (2 << 20) + 4096 * i, S) for i in range(3)]          # q, k and v of a layer
    between = [beside[0], (mats[1], zoff, S, beside[1][3], S), beside[2]]           # other rows come between
    # the first result's rows lie back to back over the bytes of token 10's Q8 row (values only: its scales stay)
    over = [(mats[0], 0, S, 10 * S, 4 * rows), (mats[1], 0, S, 2 << 20, S), (mats[2], 0, S, (2 << 20) + 4096, S)]
    assert T * 4 * rows <= cols
    for ops in (beside, between, over):
        fill()
        e.run(ops)
        got = results(ops)
        fill()
        for op in ops:
            e.run([op])
        want = results(ops)
        for g, w in zip(got, want):
            assert (g == w).all()
    e.close()


def test_chunk_without_room_for_the_attention_scratch(cuda):
    """Where the chunk attention's scratch (85 MB here) cannot be had, the chunk runs with one split of the positions: the same rows
    to the summation order, not an error. (One accumulator takes 16 products per 128 positions, 256 for these, and loses up to one
    unit of 24 bits with each: 1.6e-5 of the scale.)"""
    import torch

    from amd_c_b200 import _lib
    from amd_c_b200._lib import Op, check
    from amd_c_b200.backend import OP_ATTN, OP_ROPE_KV

    lib = _lib.load()
    nh, nkv, hd, T, n_ctx = 40, 8, 128, 256, 2048
    row, orow = (nh + 2 * nkv) * hd * 4, nh * hd * 4
    ops = (Op * 2)(Op(OP_ROPE_KV, -1, -1, 0, nh * hd, nh, 0, nh * hd * 4, (nh + nkv) * hd * 4, NONE, NONE, row, row, row, 0, 0),
                   Op(OP_ATTN, -1, -1, 0, nh * hd, 0, 0, T * row, NONE, NONE, NONE, row, orow, 0, 0, 0))
    d = _lib.EngineDesc(nh, nkv, hd, n_ctx, 1, T, 16, 1e-5, 0, 0, T * (row + orow) + 64 * T, T * (row + orow), T * (row + orow), 64, 8)
    one, zero = np.ones((n_ctx, hd // 2), np.float32), np.zeros((n_ctx, hd // 2), np.float32)
    engines = []
    for _ in range(2):
        h = C.c_void_p()
        check(lib.ie_b200_engine_create(C.byref(d), C.byref(h)))
        check(lib.ie_b200_engine_set_rope(h, one.ctypes.data_as(C.c_void_p), zero.ctypes.data_as(C.c_void_p)))
        check(lib.ie_b200_engine_set_ops(h, ops, 2, 2))
        engines.append(h)
    toks, out = np.zeros(T, np.uint32), np.zeros(T, np.uint32)

    def chunks(h):
        rng = np.random.default_rng(2)
        for pos in range(0, n_ctx, T):
            x = rng.standard_normal((T, row // 4)).astype(np.float32)
            check(lib.ie_b200_engine_write_rows(h, 0, row, 0, T, x.ctypes.data_as(C.c_void_p)))
            check(lib.ie_b200_engine_run(h, toks.ctypes.data_as(C.c_void_p), T, pos, 1, out.ctypes.data_as(C.c_void_p), None))
        y = np.zeros((T, orow // 4), np.float32)
        check(lib.ie_b200_engine_read_rows(h, T * row, orow, 0, T, y.ctypes.data_as(C.c_void_p)))
        return y

    want = chunks(engines[0])  # (also loads the kernels)
    torch.cuda.synchronize()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (48 << 20), dtype=torch.uint8, device=cuda)
    got = chunks(engines[1])
    del fill
    torch.cuda.empty_cache()
    assert np.abs(want).max() > 0.1
    assert not (got == want).all()  # one split, not several
    assert np.abs(got - want).max() <= 1.6e-5 * np.abs(want).max()
    for h in engines:
        lib.ie_b200_engine_destroy(h)


@pytest.mark.parametrize("rows,cols,T_max,T", [(3072, 8192, 384, 256), (3072, 8192, 384, 384)])
def test_gemm_workspace_holds_for_shorter_chunks(cuda, rows, cols, T_max, T):
    """The engine's GEMM workspace is sized for its longest chunk; a shorter one may split K more often and take more of it: such
    chunks run, and equal the multi-token GEMV (1e-5 of the largest output, as test_gemm_tc_matches_gemv)."""
    import torch

    from amd_c_b200 import kernels as K

    rng = np.random.default_rng(1)
    xs, ys = 40 * cols // 32, 4 * rows
    e = Engine(T_max * (xs + ys), T_max)
    m = K.Mat.from_gguf(synth.GGML_Q4_0, torch.from_numpy(np.ascontiguousarray(synth.q4_0_normal(rng, rows, cols, sigma=0.02))).to(cuda), rows, cols)
    x = _q8(torch, K, rng, T, cols, cuda)
    e.write(0, x)
    e.run([(e.add(m), 0, xs, T_max * xs, ys)], T)
    got = e.read(T_max * xs, T * rows).reshape(T, rows)
    want = K.gemv(m, torch.from_numpy(x).to(cuda)).cpu().numpy()
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    e.close()
