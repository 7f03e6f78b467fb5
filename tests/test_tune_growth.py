"""The autotuner under row-list growth: a choice stored for the earlier growth is
not read (CPU), and options that this growth has no use for are not timed (GPU)."""
import ctypes as C

import numpy as np
import pytest

from cudatree_b200 import RandomForestClassifier, _lib, tune_cache


def _shaped():
    f = RandomForestClassifier(10, max_features=7)
    f.n_samples, f.n_features, f.n_labels, f._m, f.index_bytes = 581012, 54, 7, 7, 4
    return f


def test_choices_of_the_earlier_growth_are_not_read(monkeypatch):
    monkeypatch.setenv(tune_cache.ENV, "off")
    tune_cache.clear_memory()
    shape = (581012, 54, 7, 7, 4, True, 1)
    for mode in ("batched", "plain"):
        tune_cache.put(tune_cache.key("dev", (mode, *shape)), {"scan_piece": 4096})
    f = _shaped()
    assert tune_cache.get(tune_cache.key("dev", f._shape_key("batched"))) is None
    assert tune_cache.get(tune_cache.key("dev", f._shape_key("plain"))) == {"scan_piece": 4096}
    tune_cache.clear_memory()


@pytest.mark.gpu
@pytest.mark.parametrize("misalign", [0, 2])
def test_only_options_in_use_are_timed(cuda_device, misalign):
    """Misaligned lists take list growth, whose choice may be any candidate."""
    import torch

    from . import gpu_utils as G
    rng = np.random.default_rng(4)
    y = rng.integers(0, 4, size=30000)
    x = (rng.normal(size=(30000, 8)) + y[:, None]).astype(np.float32)
    gp = G.GpuProblem(x, y, 4, 3, bootstrap=True, seed=3)
    gl = G.GpuLists(gp, 4)
    for name, si in (("si0", gl.si[0]), ("si1", gl.si[1])):
        setattr(gl.lists, name, si.data_ptr() + misalign)
    raw = [torch.zeros(4 * 2 * gp.n, dtype=torch.int32, device=G.dev()) for _ in range(5)]
    nn = torch.zeros(4, dtype=torch.int32, device=G.dev())
    tb = _lib.TreeBuffers(*[r.data_ptr() for r in raw], nn.data_ptr(), 2 * gp.n)
    ws, best, ms = C.c_size_t(), _lib.FitOptions(), C.c_float()
    _lib.call("ct_autotune_workspace_size", C.byref(gp.prob), 4, _lib.CT_FIT_BATCHED, C.byref(ws))
    work = G.dev_bytes(ws.value)
    _lib.call("ct_autotune", C.byref(gp.prob), C.byref(gl.lists), 4, _lib.CT_FIT_BATCHED, C.byref(tb),
              work.data_ptr(), ws.value, C.byref(best), C.byref(ms), G.stream())
    assert best.scan_piece in (1024, 2048, 4096) and ms.value > 0
    if misalign:
        assert best.subtree_cutoff in (0, 32, 128)
    else:
        assert best.subtree_cutoff in (0, 32)
        assert (best.part_shape, best.huge_rows, best.small_rows) == (0, 0, 0)


def _least_workspace(gp, trees, opts):
    """What list growth alone needs: an inner function of the library (no entry point returns it)."""
    fn = getattr(_lib.load(), "_ZN2ct25fit_least_workspace_bytesEPK10ct_problemjPK14ct_fit_options")
    fn.restype, fn.argtypes = C.c_size_t, [C.c_void_p, C.c_uint32, C.c_void_p]
    return fn(C.byref(gp.prob), trees, C.byref(opts))


@pytest.mark.gpu
def test_workspace_of_list_growth_is_enough(cuda_device):
    """A caller who sized the workspace for list growth alone can fit and tune."""
    import torch

    from cudatree_b200.random_forest import fetch_tree_columns
    from . import gpu_utils as G
    rng = np.random.default_rng(6)
    y = rng.integers(0, 3, size=70000)
    x = (rng.normal(size=(70000, 40)) + y[:, None] * (np.arange(40) < 5)).astype(np.float32)
    gp = G.GpuProblem(x, y, 3, 6, bootstrap=True, seed=3)
    gl = G.GpuLists(gp, 1)
    raw = [torch.zeros(2 * gp.n, dtype=torch.int32, device=G.dev()) for _ in range(5)]
    nn = torch.zeros(1, dtype=torch.int32, device=G.dev())
    tb = _lib.TreeBuffers(*[r.data_ptr() for r in raw], nn.data_ptr(), 2 * gp.n)
    opts = _lib.FitOptions(_lib.CT_FIT_BATCHED, 0, 32, 0)
    ws, tune_ws = C.c_size_t(), C.c_size_t()
    _lib.call("ct_fit_workspace_size", C.byref(gp.prob), 1, C.byref(opts), C.byref(ws))
    _lib.call("ct_autotune_workspace_size", C.byref(gp.prob), 1, _lib.CT_FIT_BATCHED, C.byref(tune_ws))
    least = _least_workspace(gp, 1, opts)
    assert least < ws.value <= tune_ws.value
    work = G.dev_bytes(ws.value)
    out = []
    for size in (ws.value, least):
        _lib.call("ct_fit", C.byref(gp.prob), C.byref(gl.lists), 0, 1, C.byref(opts), C.byref(tb), work.data_ptr(),
                  size, G.stream())
        out.append(fetch_tree_columns(tb, nn, 1, G.dev()))
    for a, b in zip([out[0][0], *out[0][1]], [out[1][0], *out[1][1]]):
        np.testing.assert_array_equal(a, b)
    best, ms = _lib.FitOptions(), C.c_float()
    _lib.call("ct_autotune", C.byref(gp.prob), C.byref(gl.lists), 1, _lib.CT_FIT_BATCHED, C.byref(tb),
              work.data_ptr(), least, C.byref(best), C.byref(ms), G.stream())
    assert ms.value > 0
