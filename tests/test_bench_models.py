"""Byte models of the benchmark's kernel figures (no GPU)."""


def test_residual_pass_bytes_count_the_elements_own_functions(small_tube):
    import bench
    mesh = small_tube.mesh
    own = sum(int(mesh.element_offsets[e + 1] - mesh.element_offsets[e]) for e in range(mesh.elements))
    assert own < 64 * mesh.elements                      # ragged: the tables' padding is not read
    read = own * 5 * 64 * 8 + mesh.elements * 64 * 11 * 8
    assert bench.residual_pass_bytes(mesh, False) == read
    assert bench.residual_pass_bytes(mesh, True) == read + mesh.elements * 72 * 64 * 4
