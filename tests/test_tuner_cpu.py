"""The tuner writes tables that the library takes, whatever shape it tries."""
import ctypes
import itertools

import build_lib
import tune


def test_tuner_tables_are_accepted(tmp_path):
    build_lib.build()
    from genericschur_gb300 import _capi
    lib = _capi.load()
    h = ctypes.c_void_p()
    lib.gs_create(ctypes.byref(h), 0)  # host-only calls work without a GPU
    path = tmp_path / "t.tsv"
    for bounds, nt in itertools.product(tune.BOUND_SETS, tune.THREADS):
        rows = [(b, nt, 0) for b in bounds]
        fp32 = [(b, nt if nt != 160 else 128, 0) for b in tune.DEFAULT_BOUNDS]
        path.write_text(tune.table_text({"real_f64": rows, "complex_f64": rows, "mixed_f32": fp32}, ["note"]))
        assert lib.gs_set_tuning(h, str(path).encode()) == 0, (bounds, nt, lib.gs_last_error(h))
    lib.gs_destroy(h)
