"""Short kernels with early launch on a stream of the caller, and under a capture of the caller's: applies of every kind
(FP64, FP32, sliced FP64; Dirichlet and hanging rows; one vector and blocks) behind the caller's own work, captured and
replayed on new values, give the bits of the context's own stream."""
import numpy as np
import pytest

import gbfe.mesh as M

pytestmark = pytest.mark.gpu


class Raw:
    def __init__(self, mv):
        self.owner = mv
        self.__cuda_array_interface__ = {"data": (mv.device_ptr(), False), "shape": mv.shape, "strides": None,
                                         "typestr": "<f8" if mv.dtype == np.float64 else "<f4", "version": 2}


@pytest.mark.parametrize("m", [1, 24, 70])
@pytest.mark.parametrize("kind", ["fp64", "fp64 hanging", "f32", "sliced"])
def test_applies_behind_and_inside_the_callers_work(kind, m):
    import torch
    from gbfe import api

    ctx = api.LinAlgOpContext(0)
    try:
        p = M.ks_box(4, 3, 8.0, 2, 4.0, 0.5, seed=11)
        if "hanging" in kind:
            p.constraints = M.add_synthetic_hanging(p.constraints, 4, 3, np.random.default_rng(1), 0.05,
                                                    inhomogeneous=True)
        dtype = np.float32 if kind == "f32" else np.float64
        basis = api.FEBasisManager.from_problem(ctx, p)
        H = api.KohnShamOperatorContextFE(basis, p.H, mixed=kind == "f32", fp64_tensor=kind == "sliced")
        ctx.set_fp64_apply(1 if kind == "sliced" else 0)
        X0 = [M.random_block(p.n_dofs, m, s).astype(dtype) for s in range(3)]
        X, Y, Z = (api.MultiVector(basis, m, dtype) for _ in range(3))
        ref = []
        for x in X0:  # Z = H H X
            X.copy_from(x)
            H.apply(X, Y)
            H.apply(Y, Z)
            ref.append(Z.numpy())
        src = [torch.from_numpy(x).cuda() for x in X0]
        tx, tz = (torch.as_tensor(Raw(v), device="cuda") for v in (X, Z))
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        with torch.cuda.stream(stream):
            for x, r in zip(src, ref):  # between the caller's copies
                tx.copy_(x)
                H.apply(X, Y)
                H.apply(Y, Z)
                got = tz.clone()
                tz.zero_()
                assert np.array_equal(got.cpu().numpy(), r)
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            graph.capture_begin(capture_error_mode="thread_local")
            H.apply(X, Y)
            H.apply(Y, Z)
            out = tz * 2.0
            graph.capture_end()
            for x, r in zip(src, ref):
                tx.copy_(x)
                graph.replay()
                assert np.array_equal(out.cpu().numpy(), 2 * r)
        stream.synchronize()
        ctx.check_status()
        ctx.set_stream(None)
    finally:
        ctx.close()


def test_noalloc_apply_under_a_capture():
    """The allocation-free apply three times in a caller's graph (each the successor of the one before)."""
    import ctypes as C

    import torch
    from gbfe import api

    ctx = api.LinAlgOpContext(0)
    try:
        p = M.ks_box(3, 3, 8.0, 2, 4.0, 0.5, seed=11)
        basis = api.FEBasisManager.from_problem(ctx, p)
        H = api.KohnShamOperatorContextFE(basis, p.H)
        X, Y = api.MultiVector(basis, 5), api.MultiVector(basis, 5)

        def apply():
            assert ctx.lib.gbfe_apply_f64_noalloc(H.h, C.c_void_p(X.device_ptr()), C.c_void_p(Y.device_ptr()), 5) == 0

        x, ref = [M.random_block(p.n_dofs, 5, s) for s in range(2)], []
        for v in x:
            X.copy_from(v)
            apply()
            ref.append(Y.numpy())
        src = [torch.from_numpy(v).cuda() for v in x]
        tx, ty = (torch.as_tensor(Raw(v), device="cuda") for v in (X, Y))
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        with torch.cuda.stream(stream):
            graph = torch.cuda.CUDAGraph()
            graph.capture_begin(capture_error_mode="thread_local")
            for _ in range(3):
                apply()
            graph.capture_end()
            for v, r in zip(src, ref):
                tx.copy_(v)
                graph.replay()
                assert np.array_equal(ty.cpu().numpy(), r)
        stream.synchronize()
        ctx.set_stream(None)
    finally:
        ctx.close()
