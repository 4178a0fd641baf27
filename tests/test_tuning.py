"""The choice of the sweep form: candidates a few percent apart must be told
apart whatever the host takes to launch a graph, and on large lattices while
the device slows down under the load.  The CUDA runtime is the model
of fake_cudart.c (a launch costs the host 4 to 12 us), so the fastest form is
known and the test runs without a GPU."""
import pytest

from test_reads import fake  # noqa: F401

# FP64 16^3 (2048 sites per parity): 16 tiles of 128 sites, 8 of 256, 4 of 2 x 256
TILES = {(128, 1): 16, (256, 1): 8, (256, 2): 4}


@pytest.mark.parametrize("calls", [[60], [16] + [5] * 10, [3] * 20, [4] * 16])
@pytest.mark.parametrize("fastest", sorted(TILES))
def test_the_fastest_form_is_chosen(fake, fastest, calls):  # noqa: F811
    """Ten passes of 7.5 us or 7.65 us: 75 against 76.5 us per sweep."""
    fake(f"""
for shape, tiles in {TILES!r}.items():
    fake.fake_cost(tiles, C.c_double(7.5 if shape == {fastest!r} else 7.65))
threads, spt, regs, wrong = C.c_int(), C.c_int(), C.c_int(), 0
for seed in range(20):
    fake.fake_seed(seed * 7919 + 1)
    p = (_lib.LceParams * 1)(Params(L=(16, 16, 16), precision="f64", seed=1).to_c())
    c = lib.lce_create_batch(p, 1)
    for n in {calls!r}:
        assert lib.lce_sweeps(c, n, 0) == 0
    assert lib.lce_get_sweep_mode(c) in (_lib.LCE_SWEEP_PASSES, _lib.LCE_SWEEP_PASSES2)
    lib.lce_get_tile_shape(c, C.byref(threads), C.byref(spt), C.byref(regs))
    wrong += (threads.value, spt.value) != {fastest!r}
    lib.lce_destroy(c)
assert wrong == 0, f"{{wrong}} of 20 contexts chose a slower form"
""")


@pytest.mark.parametrize("calls", [[40], [16] * 3, [1] * 16])
@pytest.mark.parametrize("fastest", [0, 1, 2])
def test_the_fastest_form_is_chosen_while_the_device_slows(fake, fastest, calls):  # noqa: F811
    """104 x 102 x 100, ten passes of 30 or 31 us, each sweep 1% slower than the
    one before: runs of one form after the other would favour the first."""
    tiles = [-(-104 * 102 * 100 // 2 // n) for n in (128, 256, 512)]
    fake(f"""
threads, spt, regs = C.c_int(), C.c_int(), C.c_int()
for i, tiles in enumerate({tiles!r}):
    fake.fake_cost(tiles, C.c_double(30 if i == {fastest} else 31))
for seed in range(3):
    fake.fake_seed(seed * 7919 + 1)
    p = (_lib.LceParams * 1)(Params(L=(104, 102, 100), precision="f64", seed=1).to_c())
    c = lib.lce_create_batch(p, 1)
    fake.fake_slowing(C.c_double(0.01 / 300))
    for n in {calls!r}:
        assert lib.lce_sweeps(c, n, 0) == 0
    lib.lce_get_tile_shape(c, C.byref(threads), C.byref(spt), C.byref(regs))
    assert (threads.value, spt.value) == {sorted(TILES)[fastest]!r}
    lib.lce_destroy(c)
""")
