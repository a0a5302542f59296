"""bench.py's count of kernel launches: the kernels that a wave has, and the tail pass alone of a phase without
waves."""
import bench


def test_kernels_of_a_phase():
    cart, tree, vor = "CartesianDustGrid", "TreeDustGrid", "VoronoiDustGrid"
    assert bench.phase_launches(0, cart, 500000, 10000, 0, True) == 1
    assert bench.phase_launches(20, cart, 500000, 10 ** 6, 0, False) == 80
    assert bench.phase_launches(20, cart, 500000, 10 ** 6, 0, True) == 100
    assert bench.phase_launches(200, tree, 2986747, 5 * 10 ** 8, 1 << 23, False) == 1400
    assert bench.phase_launches(30, tree, 2986747, 500000, 0, False) == 120        # too few packets to order
    assert bench.phase_launches(30, tree, 100000, 10 ** 7, 0, True) == 150         # small records
    assert bench.phase_launches(30, vor, 20000, 10 ** 6, 0, False) == 210
    assert bench.phase_launches(30, vor, 20000, 10 ** 6, 500000, False) == 120
