"""The bytes that bench.py divides by: what the kernels move, the x derivatives
that the x stage forms by itself left out, against the DRAM bytes that ncu
counted (NCU_TRAFFIC)."""
import bench


def _sizes(nx, nz, ny):
    nplanes, mz, mgalx, mgalz = nx // 2, nz - 1, 3 * nx // 2, 3 * nz // 2
    return nplanes * mz * ny, nplanes * mgalz * ny, mgalx * mgalz * ny


def test_x_stage_and_inverse_z_by_hand():
    S, Z, P = _sizes(256, 256, 65)
    # 7 input lines (all but dT/dx) read, 11 written, RHS(T) read + written
    assert bench.algo_bytes("xphys", S, Z, P, 8, 0, 0) == (7 + 11) * Z * 8 + 2 * P * 8
    # with the scalar and mu = T^sigma: 7 + 4 + 5 read, 12 written, RHS(T) and RHS(Z)
    assert bench.algo_bytes("xphys", S, Z, P, 16, 1, 1) == (16 + 12) * Z * 16 + 4 * P * 8
    assert bench.algo_bytes("zinv", S, Z, P, 8, 1, 1) == 13 * S * 8 + 16 * Z * 8
    assert bench.algo_bytes("zfwd", S, Z, P, 8, 1, 1) == bench.ALGO["zfwd"](S, Z, P, 8, 1, 1)


def test_counted_traffic_is_the_model():
    """The inputs are read once and the outputs written once: DRAM bytes within
    six percent of the model (parts of the RHS rows stay in the L2)."""
    for (name, fp64, sc, vs), t in bench.NCU_TRAFFIC.items():
        n = 768 if name == "large" else 256
        counted, ny = t["xphys"]
        model = bench.algo_bytes("xphys", *_sizes(n, n, ny), 16 if fp64 else 8, sc, vs)
        assert 0.94 < counted / model < 1.0, (name, fp64, counted / model)
