"""Short lists whose quartets' primitive quartets are split over lanes and warps, and the kernels with and
without the table of exponent pairs, against the oracle's reference-algorithm build on the CPU.

The systems cover the split's range: 128 lanes per quartet (one oxygen atom: (ss|ss) quartets of up to 4096
primitive quartets in cc-pVDZ), every smaller group as the lists grow, windows of the list that are not
full, and uncontracted shells (no split).  The engine takes the oracle's Schwartz matrix, so both screen
identically; tolerances as for the golden fixtures: 1e-10 Eh (FP64 sums of at most some 10^4 terms of size
O(10) round at 1e-12), integrals 1e-12, gradients 1e-10 Eh/bohr between two kernels on the same densities.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(name):
    from hfgpu import workloads

    if name == "O":
        return [8], np.array([[0.1, -0.2, 0.3]])
    if name == "elements":  # ten elements: over a thousand distinct exponent sums, so no table
        rng = np.random.default_rng(3)
        return list(range(1, 11)), np.array([[3.0 * k, 0.0, 0.0] for k in range(10)]) + rng.uniform(-0.4, 0.4, (10, 3))
    return workloads.water_chain(int(name), np.random.default_rng(7))


def _setup(port, basis_name, system):
    from hfgpu import basis
    from hfgpu.engine import Engine

    Z, xyz = _system(system)
    soa = basis.pack(basis_name, Z, xyz)
    e, B = Engine(soa), port.Basis(soa)
    Q = B.schwartz()
    e.set_schwartz(Q)
    return e, B, Q, Z, xyz


def _sym(n, seed, scale=0.1):
    P = np.random.default_rng(seed).standard_normal((n, n)) * scale
    return P + P.T


@pytest.mark.parametrize("basis_name,system", [("cc-pVDZ", "O"), ("cc-pVDZ", "1"), ("cc-pVDZ", "2"), ("6-311G**", "1"),
                                               ("6-31G", "3"), ("6-31G", "5"), ("STO-6G", "elements")])
@pytest.mark.parametrize("uhf", [False, True])
def test_gpu_split_lists_match_oracle(port, basis_name, system, uhf):
    e, B, Q, _, _ = _setup(port, basis_name, system)
    Da, Db = _sym(B.nao, 1), _sym(B.nao, 2)
    J, Ka, Kb, _ = e.fock(Da + Db, Da, Db if uhf else None)
    Jr, Kar, Kbr, _ = B.fock_direct(Q, Da + Db, Da, Db if uhf else None)
    for got, want in ((J, Jr), (Ka, Kar), (Kb, Kbr)):
        if want is not None:
            assert np.max(np.abs(got - want)) <= 1e-10


def test_gpu_split_matches_forced_forms(port):
    """The chunk form of the FP64 d classes, split and not, against the warp form."""
    from hfgpu.engine import FORM_AUTO, FORM_CHUNK, FORM_WARP

    e, B, Q, _, _ = _setup(port, "cc-pVDZ", "2")
    D = _sym(B.nao, 4)
    out = []
    for form in (FORM_CHUNK, FORM_WARP):
        _, avail = e.kernel_forms()
        for qc, mask in enumerate(avail):
            e.set_kernel_form(form if mask >> form & 1 else FORM_AUTO, qclass=qc)
        out.append(e.fock(2 * D, D)[:2])
    for a, b in zip(*out):
        assert np.max(np.abs(a - b)) <= 1e-10


@pytest.mark.parametrize("system", ["O", "3"])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_gpu_infinite_density_reaches_j(port, system, value):
    """No threshold: every element of J holds a multiple of the infinite element of D (0 times it is a NaN)."""
    e, B, _, _, _ = _setup(port, "6-31G", system)
    D = np.zeros((B.nao, B.nao))
    D[0, 0] = value
    J = e.fock(D, D, sthr=0.0, dthr=0.0)[0]
    assert not np.isfinite(J).any()


@pytest.mark.parametrize("atoms", [2, 12, 16, 24])
def test_gpu_infinite_density_is_infinite_in_j_and_k(atoms):
    """s functions with positive coefficients: every integral is positive, so one infinite element of D makes all of
    J and K +inf, whether a quartet has 128 lanes, some of a warp's, or one, and in a window that is not full."""
    from hfgpu import basis
    from hfgpu.engine import Engine

    xyz = np.array([(x, y, z) for x in range(4) for y in range(3) for z in range(2)][:atoms], float) * 2.0
    e = Engine(basis.pack("STO-6G", [1] * atoms, xyz))
    D = np.zeros((atoms, atoms))
    D[0, 0] = np.inf
    J, K, _, _ = e.fock(D, D, sthr=0.0, dthr=0.0)
    assert (J == np.inf).all() and (K == np.inf).all()


@pytest.mark.parametrize("shells", [(4, 4, 4, 4), (5, 4, 4, 0), (5, 5, 5, 5), (6, 5, 5, 4), (6, 5, 6, 5), (6, 6, 6, 6)])
def test_gpu_store_mode_matches_oracle(port, shells):
    """One quartet alone in store mode against the oracle's integrals, where the oracle states them (with equal
    shells it fills one of every set of equal integrals and leaves the others zero)."""
    e, B, _, _, _ = _setup(port, "cc-pVDZ", "1")  # shells: H s p, H s p, O s p d
    got, want = e.eri_block(*shells), B.eri(*shells)
    stated = want != 0.0
    assert stated.any()
    assert np.max(np.abs(got - want)[stated]) <= 1e-12 * max(1.0, np.max(np.abs(want)))


@pytest.mark.parametrize("basis_name,system", [("cc-pVDZ", "1"), ("cc-pVDZ", "2"), ("6-31G**", "3"), ("STO-6G", "elements")])
@pytest.mark.parametrize("uhf", [False, True])
def test_gpu_split_gradient_forms_agree(port, basis_name, system, uhf):
    e, B, _, Z, xyz = _setup(port, basis_name, system)
    Da, Db, W = _sym(B.nao, 1), _sym(B.nao, 2), _sym(B.nao, 3)
    g = {}
    for group_only in (False, True):
        e.set_gradient_form(group_only)
        g[group_only], _ = e.gradient(Z, xyz, Da, Db if uhf else None, W, unrestricted=uhf)
    assert np.max(np.abs(g[False] - g[True])) <= 1e-10 * max(1.0, np.max(np.abs(g[True])))
    # Translational invariance of the whole gradient.
    assert np.max(np.abs(g[False].sum(axis=0))) <= 1e-9 * max(1.0, np.max(np.abs(g[False])))


@pytest.mark.parametrize("count,kmax", [(3, 2), (24, 5)])
@pytest.mark.parametrize("precision", [0, 1])
def test_gpu_batch_lists_match_single_engines(count, kmax, precision):
    """Lists whose keys mix the bra pairs of many molecules, against one engine per molecule (mixed: the same
    FP32 quartets, summed in lists of another alignment: 1e-7)."""
    from hfgpu import basis, workloads
    from hfgpu.engine import Engine

    mols = workloads.uneven_batch(count, kmax, seed=5)
    soas = [basis.pack("6-31G", Z, xyz) for Z, xyz in mols]
    singles = [Engine(s) for s in soas]
    D = [_sym(e.nao, k, 0.05) for k, e in enumerate(singles)]
    flat = np.concatenate([d.ravel() for d in D])
    J, K, _, _ = Engine(soas).fock(2 * flat, flat, precision=precision)
    at = 0
    for e, d in zip(singles, D):
        j, k, _, _ = e.fock(2 * d, d, precision=precision)
        n2 = e.nao ** 2
        tol = 1e-10 if precision == 0 else 1e-7
        assert np.max(np.abs(J[at:at + n2] - j.ravel(order="F"))) <= tol
        assert np.max(np.abs(K[at:at + n2] - k.ravel(order="F"))) <= tol
        at += n2


@pytest.mark.parametrize("basis_name,system", [("cc-pVDZ", "2"), ("6-31G", "5")])
def test_gpu_split_graph_replay_with_another_density(port, basis_name, system):
    """A captured build sizes its grids by the eager one and reads the replay's lists on the device."""
    torch = pytest.importorskip("torch")
    e, B, Q, _, _ = _setup(port, basis_name, system)
    n = B.nao
    ins = [torch.zeros(n * n, dtype=torch.float64, device="cuda") for _ in range(2)]
    outs = [torch.zeros(n * n, dtype=torch.float64, device="cuda") for _ in range(2)]
    ptrs = dict(dD_tot=ins[0].data_ptr(), dD_alpha=ins[1].data_ptr(), J=outs[0].data_ptr(), K_alpha=outs[1].data_ptr())
    e.set_graph_mode(True)
    for seed, scale in ((1, 1e-9), (2, 0.1), (3, 1e-6)):  # few survivors when captured, many in the replay
        D = _sym(n, seed, scale)
        ins[0].copy_(torch.from_numpy(2 * D.ravel()))
        ins[1].copy_(torch.from_numpy(D.ravel().copy()))
        torch.cuda.synchronize()
        e.fock_device(ptrs)
        Jr, Kr, _, _ = B.fock_direct(Q, 2 * D, D)
        J, K = (o.cpu().numpy().reshape(n, n, order="F") for o in outs)
        assert np.max(np.abs(J - Jr)) <= 1e-10 and np.max(np.abs(K - Kr)) <= 1e-10


@pytest.mark.parametrize("basis_name,heavy,sums", [("6-31G", [6, 7, 8], 595), ("6-31G**", [6, 7, 8], 666), ("6-31G", [6, 7, 8, 9], 990)])
def test_gpu_large_exponent_table_matches_oracle(port, basis_name, heavy, sums):
    """The table of exponent pairs with several elements, up to near its limit of 1024 sums."""
    from hfgpu import basis
    from hfgpu.engine import Engine

    Z = heavy + [1]
    xyz = np.array([[2.4 * k, 0.3 * k * k, 0.0] for k in range(len(Z))])
    soa = basis.pack(basis_name, Z, xyz)
    a = np.unique(soa["alpha"])
    assert len(np.unique(a[:, None] + a[None, :])) == sums
    e, B = Engine(soa), port.Basis(soa)
    Q = B.schwartz()
    e.set_schwartz(Q)
    D = _sym(B.nao, 4)
    J, K, _, _ = e.fock(2 * D, D)
    Jr, Kr, _, _ = B.fock_direct(Q, 2 * D, D, None)
    assert np.max(np.abs(J - Jr)) <= 1e-10 and np.max(np.abs(K - Kr)) <= 1e-10
