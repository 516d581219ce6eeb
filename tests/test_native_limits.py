"""Sizes that the entry points refuse on the host, before anything is enqueued."""
import ctypes


def _cosmo(N, p, grid_size):
    c = N.HgbCosmo()
    for name, kind in N.HgbCosmo._fields_:
        if kind is ctypes.c_void_p:
            setattr(c, name, p)
    c.grid_size, c.dc_n = grid_size, 1024
    return c


def test_strain_takes_3072_frequencies_at_most(built_lib):
    from holodeck_gb300 import _native as N
    lib = N.load()
    p = 256   # a non-null address that is never dereferenced: the checks return first
    c = _cosmo(N, p, 50)
    for nf in (3073, 1 << 20):
        rc = lib.hgb_char_strain_sq(p, 3, p, 3, 3, p, nf, p, 1.0, ctypes.byref(c), p, None, None)
        assert rc == N.HGB_ERR_INVALID_ARGUMENT
        rc = lib.hgb_number_and_strain(p, p, 3, p, 3, p, 3, p, p, nf, p, p, 1.0, ctypes.byref(c), p, p, None, None)
        assert rc == N.HGB_ERR_INVALID_ARGUMENT


def test_walk_tables_of_one_cell_stay_below_200_kb(built_lib):
    from holodeck_gb300 import _native as N
    lib = N.load()
    p = 256
    for grid_size, steps, nf in ((50, 5100, 1), (50, 4900, 1000)):   # 32 grid_size + 8 nf + 40 steps bytes
        c = _cosmo(N, p, grid_size)
        for ascending in (0, 1):
            rc = lib.hgb_dbn_2pwl_phase(p, nf, ascending, 1.0, steps, p, 1.0, -1.0, 2.5, p, p, 1, p, 1, p, 1, p,
                                        ctypes.byref(c), p, p, 1, None)
            assert rc == N.HGB_ERR_INVALID_ARGUMENT
