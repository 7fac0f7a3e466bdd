"""Edges of the sizes at which the device path changes kernels or splits, against the oracle."""
import numpy as np
import pytest
import torch

from fourierd3_b200 import D3Model, FourierD3, _native, neighbour_list, structures
from oracle.neighbours import neighbour_list_cells
from oracle.reference_port import OracleFourierD3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_atoms", [1, 33, 250, 264, 2300])
def test_neighbours_of_bins_from_one_to_hundreds_of_atoms(cuda_device, n_atoms):
    # 2 x 2 x 2 bins of 6.05 A: segments of the counting sort below, at and far beyond one warp
    rng = np.random.default_rng(n_atoms)
    cell = np.diag([12.1, 12.1, 12.1])
    pos = rng.random((n_atoms, 3)) @ cell
    i, j, s = neighbour_list(torch.tensor(pos, device=cuda_device), cell, 6.0)
    got = torch.cat((i[:, None], j[:, None], s.to(torch.int64)), 1).cpu().numpy()
    ri, rj, rs = neighbour_list_cells(pos, cell, 6.0)
    want = np.concatenate((ri[:, None], rj[:, None], rs), 1)
    assert np.all(np.diff(got[:, 0]) >= 0)
    assert np.array_equal(got[np.lexsort(got.T[::-1])], want[np.lexsort(want.T[::-1])])


def _against_oracle(device, pos, cell, numbers, precision, tol, **kw):
    o = OracleFourierD3(numbers, cell, **kw)
    i, j, s = neighbour_list_cells(pos, cell, 6.0)
    e_ref, f_ref, s_ref = o.calculate(pos, cell, edges=(np.stack([i, j]), s))
    e, f, st = D3Model(numbers, cell, precision=precision, device=device, **kw)(pos, cell)
    assert abs(float(e) - e_ref) <= tol[0] * abs(e_ref)
    assert np.abs(f.cpu().numpy() - f_ref).max() <= tol[1]
    assert np.abs(st.cpu().numpy() - s_ref).max() <= tol[2]


# the tolerances of the two forms against the oracle (energy relative, eV/A, eV/A^3)
TOL = {"fp64": (1e-10, 1e-8, 1e-9), "mixed": (1e-6, 1e-4, 1e-6)}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("edge,n_atoms", [(1.9, 1), (2.9, 3), (5.2, 14), (12.2, 60), (12.2, 420), (19.0, 500)])
def test_cn_stage_from_image_only_cells_to_bins_beyond_the_stage(cuda_device, edge, n_atoms, precision):
    # 1.9 A: more neighbour bins than the table holds (traversal of global memory); 2.9 and 5.2 A: every
    # candidate is an image of one bin; 420 atoms in 12.2 A: 27 bins of 52, pieces of the stage and
    # atoms with more pairs than the record holds; 19 A: several CTAs per bin
    rng = np.random.default_rng(n_atoms)
    cell = np.diag([edge, edge, edge]) + np.triu(np.full((3, 3), 0.03 * edge), 1)
    m = int(np.ceil(n_atoms ** (1 / 3)))
    grid = rng.permutation(m ** 3)[:n_atoms]
    frac = (np.stack(np.unravel_index(grid, (m, m, m)), 1) + rng.uniform(0.4, 0.6, (n_atoms, 3))) / m
    numbers = rng.choice([1, 6, 8], n_atoms)
    _against_oracle(cuda_device, frac @ cell, cell, numbers, precision, TOL[precision], method="spme",
                    mesh_spacing=1.2, interpolation_nodes=4, c6tol=1.0, r_cut=6.0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_atoms", [2047, 2048, 2049])
def test_preparation_in_one_cta_and_in_several_launches(cuda_device, n_atoms, precision):
    # the one-CTA sort takes up to 2,048 atoms; same density, one atom more or less
    pos, cell, numbers = structures.hcno_box(seed=5, n_atoms=n_atoms)
    _against_oracle(cuda_device, pos, cell, numbers, precision, TOL[precision], method="pme", mesh_spacing=1.2,
                    interpolation_nodes=4, c6tol=1.0, r_cut=6.0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_atoms,z_max,k_cutoff", [(1, 1, 2.0), (33, 8, 3.1), (130, 30, 2.2)])
def test_ewald_sums_over_tiles_rows_and_many_species(cuda_device, n_atoms, z_max, k_cutoff, precision):
    # odd and even Miller boxes, one species and dozens (several filter tiles, more than 8 ranks or not)
    pos, cell, numbers = structures.random_box(seed=n_atoms, n_atoms=n_atoms, z_max=z_max)
    _against_oracle(cuda_device, pos, cell, numbers, precision, TOL[precision], method="ewald", k_cutoff=k_cutoff,
                    c6tol=0.05, r_cut=6.0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order,z_max,c6tol", [(6, 8, 1.0), (7, 3, 1.0), (5, 40, 0.05), (8, 25, 0.2)])
def test_gather_of_any_order_and_rank_count(cuda_device, order, z_max, c6tol, precision):
    # rank chunks with and without a remainder, runs of every offset and the wrapped ones
    pos, cell, numbers = structures.random_box(seed=order, n_atoms=70, z_max=z_max)
    _against_oracle(cuda_device, pos, cell, numbers, precision, TOL[precision], method="spme", mesh_spacing=1.2,
                    interpolation_nodes=order, c6tol=c6tol, r_cut=6.0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("lengths", [(24.0, 8.0, 8.0), (24.0, 8.0, 16.0), (24.0, 16.0, 8.0), (24.0, 32.0, 32.0), (36.0, 70.0, 8.0),
                                     (24.0, 8.0, 70.0), (40.0, 66.0, 32.0), (24.0, 66.0, 67.0), (24.0, 130.0, 24.0),
                                     (24.0, 24.0, 130.0), (24.0, 130.0, 66.0)])
def test_plane_transforms_of_every_length_agree_with_cufft(cuda_device, lengths, precision):
    # planes from 16 x 16 points to the largest that a CTA holds and beyond (cuFFT then), against the 3D transforms
    rng = np.random.default_rng(int(sum(lengths)))
    cell = np.diag(lengths)
    numbers = rng.choice([8, 14], 90)
    pos = rng.random((90, 3)) @ cell
    m = D3Model(numbers, cell, precision=precision, device=cuda_device, method="spme", mesh_spacing=1.2,
                interpolation_nodes=4, r_cut=6.0)
    m.engine.set_tuning(fft_x=0)
    e0, f0, s0 = (t.clone() for t in m(pos, cell))
    m.engine.set_tuning(fft_x=1)
    e, f, s = m(pos, cell)
    tol_e, tol_f = (1e-12, 1e-10) if precision == "fp64" else (2e-6, 1e-5)
    assert abs(float(e) - float(e0)) <= tol_e * abs(float(e0))
    assert (f - f0).abs().max().item() <= tol_f
    assert (s - s0).abs().max().item() <= tol_f


@pytest.mark.parametrize("lengths,z_max,c6tol", [((8.0, 8.0, 8.0), 4, 1.0), ((8.0, 24.0, 8.0), 1, 1.0),
                                                 ((16.0, 8.0, 16.0), 2, 1.0), ((32.0, 8.0, 8.0), 4, 0.05),
                                                 ((66.0, 16.0, 8.0), 3, 1.0), ((130.0, 8.0, 8.0), 4, 1.0)])
def test_float64_x_pass_of_every_length(cuda_device, lengths, z_max, c6tol):
    # nx = 16 to 256, one to four species, sheared (the partner of a self-conjugate k has another length),
    # each pencil width, against the 3D transforms around the separate filter
    rng = np.random.default_rng(int(sum(lengths)) + z_max)
    cell = np.diag(lengths) + np.triu(np.full((3, 3), 1.1), 1)
    numbers = rng.integers(1, z_max + 1, 60)
    pos = rng.random((60, 3)) @ cell
    m = D3Model(numbers, cell, precision="fp64", device=cuda_device, method="spme", mesh_spacing=1.2,
                interpolation_nodes=4, c6tol=c6tol, r_cut=6.0)
    m.engine.set_tuning(fft_x=0)
    e0, f0, s0 = (t.clone() for t in m(pos, cell))
    for kz in (-1, 1, 2, 4):
        m.engine.set_tuning(fft_x=1, xpencil=kz)
        e, f, s = m(pos, cell)
        assert abs(float(e) - float(e0)) <= 1e-12 * abs(float(e0))
        assert (f - f0).abs().max().item() <= 1e-10 * max(1.0, f0.abs().max().item())
        assert (s - s0).abs().max().item() <= 1e-10 * max(1.0, s0.abs().max().item())


@pytest.mark.parametrize("n_species,c6tol", [(15, 1.0), (16, 30.0), (17, 1.0), (40, 1.0), (41, 30.0), (43, 1.0)])
def test_many_species_filter_agrees_with_the_tiled_one(cuda_device, n_species, c6tol):
    # below its range, whole and ragged 4 x 4 blocks, both tile widths, up to 4 and up to 8 ranks, a sheared cell
    rng = np.random.default_rng(n_species)
    numbers = np.concatenate((np.arange(1, n_species + 1), rng.integers(1, n_species + 1, 60)))
    cell = np.diag([9.0, 12.0, 10.0]) + np.triu(np.full((3, 3), 0.9), 1)
    pos = rng.random((len(numbers), 3)) @ cell
    m = D3Model(numbers, cell, precision="mixed", device=cuda_device, method="spme", mesh_spacing=1.2,
                interpolation_nodes=4, c6tol=c6tol, r_cut=6.0)
    e, f, s = (t.clone() for t in m(pos, cell))
    m.engine.set_tuning(filter_kt=4)
    e0, f0, s0 = m(pos, cell)
    assert abs(float(e) - float(e0)) <= 2e-6 * abs(float(e0))
    assert (f - f0).abs().max().item() <= 1e-5 * max(1.0, f0.abs().max().item())
    assert (s - s0).abs().max().item() <= 1e-5 * max(1.0, s0.abs().max().item())


@pytest.mark.parametrize("n_atoms,n_edges", [(5, 1), (700, 3), (40, 255), (40, 257), (300, 9000)])
def test_edge_lists_sorted_by_source_or_in_any_order(cuda_device, n_atoms, n_edges):
    # the two ways to the source segments: atoms without edges first, last and in runs, blocks of 256 edges
    rng = np.random.default_rng(n_edges)
    cell = torch.tensor(np.diag([26.0, 30.0, 28.0]), device=cuda_device)
    numbers = rng.choice([8, 14], n_atoms)
    pos = torch.tensor(rng.random((n_atoms, 3)) * 26.0, device=cuda_device)
    active = np.arange(n_atoms // 3, n_atoms - n_atoms // 5)
    src = torch.tensor(np.sort(rng.choice(active, n_edges)), device=cuda_device)
    dst = torch.tensor(rng.choice(n_atoms, n_edges), device=cuda_device)
    shift = torch.tensor(rng.normal(size=(n_edges, 3)) * 3.0, device=cuda_device)
    m = FourierD3(numbers, cell.cpu().numpy(), dtype=torch.float64, device=cuda_device, verbose=False,
                  method="spme", mesh_spacing=2.0, interpolation_nodes=4, r_cut=12.0)

    def run(order):
        p = pos.clone().requires_grad_()
        sh = shift[order].clone().requires_grad_()
        e = m(p, torch.stack((src[order], dst[order])), sh)
        e.backward()
        g = torch.empty_like(shift)
        g[order] = sh.grad
        return e.detach(), p.grad, g

    e0, p0, g0 = run(torch.arange(n_edges, device=cuda_device))
    for _ in range(2):
        e, p, g = run(torch.tensor(rng.permutation(n_edges), device=cuda_device))
        assert abs(float(e - e0)) <= 1e-12 * abs(float(e0))
        assert (p - p0).abs().max().item() <= 1e-12 * max(1e-3, p0.abs().max().item())
        assert (g - g0).abs().max().item() <= 1e-12 * max(1e-3, g0.abs().max().item())


@pytest.mark.parametrize("spacing,z", [(0.16, 55), (0.4, 55), (1.2, 1), (1.2, 55), (4.0, 30)])
def test_float64_green_function_from_tables(cuda_device, spacing, z):
    # from the smallest |k| R to exponentials below 1e-20: register filter and x-pass (tables) against the tiled filter
    rng = np.random.default_rng(z)
    cell = np.diag([7.0, 8.0, 7.5]) + np.triu(np.full((3, 3), 0.6), 1)
    numbers = rng.choice([1, z], 20)
    pos = rng.random((20, 3)) @ cell
    m = D3Model(numbers, cell, precision="fp64", device=cuda_device, method="spme", mesh_spacing=spacing,
                interpolation_nodes=4, c6tol=1.0, r_cut=6.0)
    m.engine.set_tuning(fft_x=0, filter_kt=4)
    e0, f0, s0 = (t.clone() for t in m(pos, cell))
    for fft_x in (0, 1):
        m.engine.set_tuning(fft_x=fft_x, filter_kt=-1)
        e, f, s = m(pos, cell)
        assert abs(float(e) - float(e0)) <= 1e-12 * abs(float(e0))
        assert (f - f0).abs().max().item() <= 1e-10 * max(1.0, f0.abs().max().item())
        assert (s - s0).abs().max().item() <= 1e-10 * max(1.0, s0.abs().max().item())


@pytest.mark.parametrize("n_atoms", [420, 3000, 17000])
def test_dense_bins_of_the_mixed_form_stay_in_float64(cuda_device, n_atoms):
    # more than 768 candidates per bin: the mixed form takes such bins in float64, and the direct sum adds
    # nothing but float64 to them, so that both forms differ by the order of their sums alone: some 1e3 terms of
    # 1e-16, up to ten times the largest force each, 1e-12. 420 atoms: pieces of the stage, records that overflow;
    # 17,000: the records in a launch of their own
    if n_atoms == 420:
        rng = np.random.default_rng(n_atoms)
        cell = np.diag([12.2, 12.2, 12.2]) + np.triu(np.full((3, 3), 0.4), 1)
        grid = rng.permutation(512)[:n_atoms]
        pos = (np.stack(np.unravel_index(grid, (8, 8, 8)), 1) + rng.uniform(0.4, 0.6, (n_atoms, 3))) / 8 @ cell
        numbers = rng.choice([1, 6, 8], n_atoms)
    else:
        pos, cell, numbers = structures.hcno_box(seed=7, n_atoms=n_atoms)
    out = [D3Model(numbers, cell, precision=p, device=cuda_device, method="spme", mesh_spacing=2.4,
                   interpolation_nodes=4, c6tol=1.0, r_cut=6.0).direct(pos, cell, 8.0) for p in ("fp64", "mixed")]
    for want, got in zip(*out):
        assert (got - want).abs().max().item() <= 1e-12 * want.abs().max().item()


@pytest.mark.parametrize("k_cutoff", [1.0, 4.0, 10.0])
def test_an_ewald_workspace_made_for_more_atoms_serves_fewer(cuda_device, k_cutoff):
    # through the counts at which the sums change their number of chunks, and one call in a workspace for more
    pos, cell, numbers = structures.random_box(seed=3, n_atoms=40, z_max=8)
    m = D3Model(numbers, cell, precision="fp64", device=cuda_device, method="ewald", k_cutoff=k_cutoff, r_cut=6.0)
    size = [m.engine.workspace_bytes(n, cell, 6.0) for n in (*range(1, 1500), *range(74000, 77000), 151551, 151552, 151553)]
    assert all(a <= b for a, b in zip(size, size[1:]))
    e, f, s = (t.clone() for t in m(pos, cell))
    work = torch.empty(m.engine.workspace_bytes(41, cell, 6.0), dtype=torch.uint8, device=cuda_device)
    got = m.engine.energy_forces_stress(torch.tensor(pos, device=cuda_device), cell, 6.0, work=work)
    assert all(torch.equal(a, b) for a, b in zip(got, (e, f, s)))


def _box(lengths, numbers, seed):
    rng = np.random.default_rng(seed)
    cell = np.diag(lengths) + np.triu(np.full((3, 3), 0.3), 1)
    return rng.random((len(numbers), 3)) @ cell, cell


def _settable(t):
    # 0 stands for "does not apply" in these, and is not a setting
    return {k: v for k, v in t.items() if v != 0 or k not in ("xpencil", "xq", "xranks")}


@pytest.mark.parametrize("precision,method,lengths,n_species", [
    ("fp64", "spme", (36.0, 36.0, 36.0), 2), ("fp64", "spme", (8.0, 16.0, 8.0), 3), ("fp64", "pme", (24.0, 8.0, 140.0), 2),
    ("mixed", "spme", (36.0, 36.0, 36.0), 2), ("mixed", "spme", (36.0, 8.0, 36.0), 4), ("mixed", "pme", (16.0, 16.0, 16.0), 2),
    ("mixed", "spme", (36.0, 140.0, 140.0), 1), ("mixed", "ewald", (9.0, 9.0, 9.0), 2), ("mixed", "spme", (9.0, 12.0, 10.0), 20),
    ("mixed", "spme", (9.0, 12.0, 10.0), 10), ("fp64", "spme", (9.0, 12.0, 10.0), 20)])
def test_settings_read_back_and_set_again_change_no_kernel(cuda_device, precision, method, lengths, n_species):
    numbers = np.concatenate((np.arange(1, n_species + 1), np.random.default_rng(4).integers(1, n_species + 1, 60)))
    pos, cell = _box(lengths, numbers, 5)

    def run(tuning):
        m = D3Model(numbers, cell, precision=precision, device=cuda_device, method=method, mesh_spacing=1.2,
                    interpolation_nodes=4, r_cut=6.0)
        if tuning is not None:
            m.engine.set_tuning(**_settable(tuning))
        launches = _native.launch_count()
        out = [t.clone() for t in m(pos, cell)]
        return m.engine.tuning(), _native.launch_count() - launches, out

    tuning, launches, out = run(None)
    again = run(tuning)
    assert again[0] == tuning and again[1] == launches
    assert all(torch.equal(a, b) for a, b in zip(again[2], out))


@pytest.mark.parametrize("sources", [(100000, 100009), (0, 1), (199998, 199999)])
def test_sorted_edges_on_a_few_of_many_atoms(cuda_device, sources):
    # 200,000 atoms, two of them with edges: the same results as in descending order, and no slower (the segment
    # starts of the atoms without edges are one run of stores; half as long again is left for the timer)
    n = 200000
    rng = np.random.default_rng(8)
    cell = torch.tensor(np.diag([230.0] * 3), device=cuda_device)
    numbers = rng.choice([8, 14], n)
    pos = torch.tensor(rng.random((n, 3)) * 230.0, device=cuda_device)
    m = FourierD3(numbers, cell.cpu().numpy(), dtype=torch.float64, device=cuda_device, verbose=False, method="spme",
                  mesh_spacing=8.0, interpolation_nodes=4, r_cut=12.0)
    edges = torch.tensor([sources, sources[::-1]], device=cuda_device)
    shift = torch.tensor([[1.0, 2.0, 3.0], [-1.0, -2.0, -3.0]], dtype=torch.float64, device=cuda_device)
    shift -= pos[edges[1]] - pos[edges[0]]
    m._eng.profile(True)
    out, ms = [], []
    for order in ([0, 1], [1, 0]):
        times = []
        for _ in range(6):
            got = m._eng.energy_edges(pos, cell, edges[:, order], shift[order], True)
            times.append(m._eng.stage_times()["cn_c6"])
        out.append((got[0].clone(), got[1].clone(), got[2][order].clone(), got[3].clone()))
        ms.append(np.median(times[1:]))
    assert all(torch.equal(a, b) for a, b in zip(*out))
    assert ms[0] <= 1.5 * ms[1]


@pytest.mark.parametrize("mesh,z_max,c6tol,want", [
    ((64, 64, 64), 4, 1.0, (1, 4)), ((64, 64, 32), 4, 1.0, (1, 2)), ((128, 64, 16), 4, 1.0, (1, 1)),
    ((32, 256, 32), 2, 1.0, (1, 4)), ((256, 32, 16), 2, 1.0, (1, 1)),
    ((256, 64, 64), 8, 1.0, (0, None)), ((64, 256, 256), 2, 1.0, (0, None))])
def test_float64_x_pass_by_default_where_it_was_measured_faster(cuda_device, mesh, z_max, c6tol, want):
    # the pencil width that fills the chip, and the separate filter where one pencil at a time fits an SM or the planes
    # are cuFFT's
    lengths = [(0.8 * n - 1.0) * 0.6 for n in mesh]
    numbers = np.concatenate(([1, 6, 7, 8] if z_max == 8 else np.arange(1, z_max + 1), [1] * 20))
    m = D3Model(numbers, np.diag(lengths), precision="fp64", device=cuda_device, method="spme", mesh_spacing=1.2,
                interpolation_nodes=4, c6tol=c6tol, r_cut=6.0)
    assert tuple(m.mesh) == mesh
    t = m.engine.tuning()
    assert t["fft_x"] == want[0] and (want[1] is None or t["xpencil"] == want[1]), (t, m.setup.n_rank)


def _launches(m, pos, cell, **knobs):
    m.engine.set_tuning(**knobs)
    before = _native.launch_count()
    m(pos, cell)
    return _native.launch_count() - before


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("mesh", [(64, 16, 16), (64, 16, 32), (64, 32, 16), (64, 64, 64), (64, 128, 16), (64, 16, 128),
                                  (128, 128, 64), (64, 128, 128), (64, 256, 64), (64, 64, 256), (64, 256, 128),
                                  (64, 8, 16)])
def test_planes_that_fit_a_cta_are_the_librarys_own(cuda_device, mesh, precision):
    # the x-pass in place of the filter, and a launch each way for the planes unless they are cuFFT's
    lengths = [(0.8 * n - 1.0) * 0.6 for n in mesh]
    numbers = np.array([8, 14] * 20)
    pos, _ = _box(lengths, numbers, 9)
    cell = np.diag(lengths)
    m = D3Model(numbers, cell, precision=precision, device=cuda_device, method="spme", mesh_spacing=1.2,
                interpolation_nodes=4, r_cut=6.0)
    assert tuple(m.mesh) == mesh
    separate = _launches(m, pos, cell, fft_x=0)
    fused = _launches(m, pos, cell, fft_x=1)
    assert m.engine.tuning()["fft_x"] == 1
    own = min(mesh[1:]) >= 16 and mesh[1] * mesh[2] <= (128 * 128 if precision == "fp64" else 128 * 256)
    assert fused - separate == (2 if own else 0)


@pytest.mark.parametrize("lengths,z_max,c6tol", [((8.0, 8.0, 8.0), 4, 1.0), ((8.0, 24.0, 8.0), 1, 1.0),
                                                 ((16.0, 8.0, 16.0), 2, 1.0), ((32.0, 8.0, 8.0), 4, 0.05),
                                                 ((66.0, 16.0, 8.0), 3, 1.0), ((130.0, 8.0, 8.0), 4, 1.0)])
def test_float64_x_pass_takes_every_length_and_width(cuda_device, lengths, z_max, c6tol):
    # the cases of test_float64_x_pass_of_every_length run the x-pass, at the width asked for or the widest that fits
    rng = np.random.default_rng(int(sum(lengths)) + z_max)
    cell = np.diag(lengths) + np.triu(np.full((3, 3), 1.1), 1)
    m = D3Model(rng.integers(1, z_max + 1, 60), cell, precision="fp64", device=cuda_device, method="spme",
                mesh_spacing=1.2, interpolation_nodes=4, c6tol=c6tol, r_cut=6.0)
    got = []
    for kz in (1, 2, 4):
        m.engine.set_tuning(fft_x=1, xpencil=kz)
        t = m.engine.tuning()
        assert t["fft_x"] == 1 and t["xpencil"] <= kz
        got.append(t["xpencil"])
    assert got == [min(kz, got[2]) for kz in (1, 2, 4)] and got[2] >= 2


def test_float64_green_function_of_a_coarse_mesh_in_the_x_pass(cuda_device):
    # the longest spacing of test_float64_green_function_from_tables on a mesh that the x-pass takes (16^3)
    rng = np.random.default_rng(30)
    cell = np.diag([15.0, 16.0, 15.5]) + np.triu(np.full((3, 3), 0.6), 1)
    numbers = rng.choice([1, 30], 60)
    pos = rng.random((60, 3)) @ cell
    m = D3Model(numbers, cell, precision="fp64", device=cuda_device, method="spme", mesh_spacing=4.0,
                interpolation_nodes=4, c6tol=1.0, r_cut=6.0)
    m.engine.set_tuning(fft_x=0, filter_kt=4)
    e0, f0, s0 = (t.clone() for t in m(pos, cell))
    m.engine.set_tuning(fft_x=1, filter_kt=-1)
    assert m.engine.tuning()["fft_x"] == 1
    e, f, s = m(pos, cell)
    assert abs(float(e) - float(e0)) <= 1e-12 * abs(float(e0))
    assert (f - f0).abs().max().item() <= 1e-10 * max(1.0, f0.abs().max().item())
    assert (s - s0).abs().max().item() <= 1e-10 * max(1.0, s0.abs().max().item())


@pytest.mark.parametrize("n_species,c6tol,runs", [(15, 1.0, False), (16, 30.0, True), (40, 1.0, True), (41, 1.0, True),
                                                  (64, 30.0, True), (64, 1.0, True)])
def test_many_species_filter_up_to_the_most_it_takes(cuda_device, n_species, c6tol, runs):
    # which kernel filters by default (no k-tile in effect: the many-species one), and 64 species against the tiled one
    rng = np.random.default_rng(n_species)
    numbers = np.concatenate((np.arange(1, n_species + 1), rng.integers(1, n_species + 1, 60)))
    cell = np.diag([9.0, 12.0, 10.0]) + np.triu(np.full((3, 3), 0.9), 1)
    pos = rng.random((len(numbers), 3)) @ cell
    m = D3Model(numbers, cell, precision="mixed", device=cuda_device, method="spme", mesh_spacing=1.2,
                interpolation_nodes=4, c6tol=c6tol, r_cut=6.0)
    assert m.setup.n_rank <= 8 and (m.engine.tuning()["filter_kt"] == -1) == runs
    e, f, s = (t.clone() for t in m(pos, cell))
    m.engine.set_tuning(filter_kt=2)
    assert m.engine.tuning()["filter_kt"] == 2
    e0, f0, s0 = m(pos, cell)
    assert abs(float(e) - float(e0)) <= 2e-6 * abs(float(e0))
    assert (f - f0).abs().max().item() <= 1e-5 * max(1.0, f0.abs().max().item())
    assert (s - s0).abs().max().item() <= 1e-5 * max(1.0, s0.abs().max().item())


@pytest.mark.parametrize("precision,method,cnfunc", [("fp64", "spme", "smooth_cut"), ("mixed", "spme", "smooth_cut"),
                                                     ("fp64", "pme", "d4"), ("mixed", "ewald", "smooth_cut")])
def test_a_captured_call_keeps_its_host_cell_and_takes_new_positions(cuda_device, precision, method, cnfunc):
    # without a device copy of the cell it travels with the launches, so that a graph holds the cell of its capture
    pos, cell, numbers = structures.hcno_box(seed=9, n_atoms=120)
    m = D3Model(numbers, cell, precision=precision, device=cuda_device, method=method, cnfunc=cnfunc, mesh_spacing=1.2,
                interpolation_nodes=4, c6tol=1.0, r_cut=6.0)
    x = torch.tensor(pos, device=cuda_device)
    moved = torch.tensor(pos + 0.1 * np.random.default_rng(1).normal(size=pos.shape), device=cuda_device)
    want = [[t.clone() for t in m.engine.energy_forces_stress(p, cell, 6.0)] for p in (x, moved)]
    host_cell = np.array(cell)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = m.engine.energy_forces_stress(x, host_cell, 6.0)
    host_cell *= 1.1
    for p, w in zip((torch.tensor(pos, device=cuda_device), moved), want):
        x.copy_(p)
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, w))


@pytest.mark.parametrize("precision,element,mesh,want", [
    ("mixed", 8, (128, 128, 128), 2), ("mixed", 8, (64, 256, 256), 0), ("mixed", 1, (64, 256, 256), 2),
    ("fp64", 8, (64, 64, 64), 1), ("fp64", 8, (64, 128, 64), 1), ("fp64", 8, (64, 64, 256), 0), ("fp64", 1, (256, 64, 64), 1)])
def test_x_pass_by_default_with_one_species(cuda_device, precision, element, mesh, want):
    # three ranks (oxygen) leave a rank group partly empty, two (hydrogen) do not; large planes in float64
    lengths = [(0.8 * n - 1.0) * 0.6 for n in mesh]
    m = D3Model(np.full(20, element), np.diag(lengths), precision=precision, device=cuda_device, method="spme",
                mesh_spacing=1.2, interpolation_nodes=4, c6tol=0.01 if element == 8 else 1.0, r_cut=6.0)
    assert tuple(m.mesh) == mesh and m.setup.n_rank == (3 if element == 8 else 2)
    assert m.engine.tuning()["fft_x"] == want


@pytest.mark.parametrize("precision,n_atoms", [("mixed", 32000), ("mixed", 90000), ("mixed", 400000), ("fp64", 37000),
                                               ("fp64", 400000)])
def test_column_spread_of_full_and_overfull_chunks(cuda_device, precision, n_atoms):
    # 128^3, chunks of 8 z-tiles: nearly as full as the stage, several times as full, and with single tiles that
    # overflow it. The results of chunks of one tile and of the per-tile kernel, to rounding; where the stage holds the
    # chunk, in about the time of chunks of one tile (a stage of 226 float atoms, of 250 before, did not: 2.1 times)
    lengths = [(n_atoms / 0.07) ** (1 / 3)] * 3
    rng = np.random.default_rng(n_atoms)
    m1 = int(np.ceil(n_atoms ** (1 / 3)))
    grid = np.stack(np.unravel_index(np.sort(rng.permutation(m1**3)[:n_atoms]), (m1,) * 3), 1)
    cell = np.diag(lengths)
    pos = torch.tensor((grid + rng.uniform(0.2, 0.8, grid.shape)) / m1 @ cell, device=cuda_device)
    numbers = np.where(grid.sum(1) % 2 == 0, 8, 14)
    m = D3Model(numbers, cell, precision=precision, device=cuda_device, method="spme", mesh_spacing=lengths[0] / 51.2,
                interpolation_nodes=5, c6tol=1.0, r_cut=6.0)
    assert tuple(m.mesh) == (128, 128, 128) and m.setup.n_rank == 4
    m.engine.profile(True)
    out, ms = {}, {}
    for zc in (8, 1, 0):
        m.engine.set_tuning(spread_zc=zc)
        assert m.engine.tuning()["spread_zc"] == zc
        times = []
        for _ in range(6):
            out[zc] = [t.clone() for t in m(pos, cell)]
            times.append(m.engine.stage_times()["spread"])
        ms[zc] = np.median(times[1:])
    e_tol, f_tol = (1e-12, 1e-10) if precision == "fp64" else (2e-6, 1e-5)
    for zc in (1, 0):
        for k, tol in enumerate((e_tol, f_tol, f_tol)):
            scale = out[zc][k].abs().max().item()
            assert (out[8][k] - out[zc][k]).abs().max().item() <= tol * (scale if k == 0 else max(1.0, scale))
    if n_atoms == 32000:
        assert ms[8] <= 1.5 * ms[1]
