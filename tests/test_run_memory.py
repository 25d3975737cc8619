"""What an electrified run holds on the device beyond a two-moment run (host arithmetic; no GPU)."""
from meteolab_gb300 import build


def test_the_lightning_holds_only_what_its_kernels_use():
    """Per node four FP64 arrays (the charge, its potential, the growth front's two) and eight 32-bit ones; per mode of the
    potential's solve its spectrum and three coefficients; the channel, tables and partial sums beside them are small."""
    build.build()
    from meteolab_gb300 import runtime
    from meteolab_gb300.grid import DEFAULT_GRID, create_grid
    from meteolab_gb300.scenarios import Switches
    g = create_grid(DEFAULT_GRID)
    electrified, rain2 = runtime.run_bytes(g, Switches(lightning=1)), runtime.run_bytes(g, Switches(rain_moments=2))
    solve = (g.nz - 2) * (g.nx // 2 + 1) * g.ny * (16 + 3 * 8)
    assert electrified - rain2 <= g.n * (4 * 8 + 8 * 4) + solve + 4 * 3000 * 8 + 64 * 1024
