"""Assembly kernels at their edges: the device pattern's register sorts (32, 64,
128 and 256 contributions a row, columns too far away for the 32-bit key, rows
left to the shared-memory sort), the multi-block scans, the device layout of the
sliced ELL and its packing, each against the host builder."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ("rowptr", "col", "slot_ptr", "slot_src", "diag")


def _fans(k, degrees, rng):
    """Elements of k nodes whose i-th hub node has degrees[i] of them; every node is in one."""
    out, n = [], len(degrees)
    for hub, deg in enumerate(degrees):
        rim = np.arange(n, n + max(deg, k))
        n += len(rim)
        for i in range(deg):
            el = [hub] + [int(rim[(i + j) % len(rim)]) for j in range(k - 1)]
            out.append(rng.permutation(el))
        out.append(rim[:k])                                # short fans: every rim node has an element
        out.extend(rim[j: j + k] if j + k <= len(rim) else rim[-k:] for j in range(k, len(rim), k))
    return rng.permutation(np.array(out, dtype=np.int32)), n


def _equal(el, n, cuda):
    from torchcor_b200.core.assemble import build_pattern, build_pattern_device
    h = build_pattern(el, n)
    g = build_pattern_device(torch.from_numpy(el).to(cuda), n)
    assert g.nnz == h.nnz
    for name in NAMES:
        assert np.array_equal(g.host(name), h.host(name)), name
    return h


@pytest.mark.parametrize("k,degrees", [
    (4, [1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 200, 255]),
    (3, [1, 9, 10, 11, 20, 21, 22, 31, 32, 33, 63, 64, 65, 100, 340]),
])
def test_rows_of_every_sort(lib, cuda, k, degrees):
    el, n = _fans(k, degrees, np.random.default_rng(k))
    _equal(el, n, cuda)


@pytest.mark.parametrize("k,shift,inplace", [(4, 0, False), (4, 1, False), (4, 1, True), (3, 1, False)])
def test_contributions_beside_and_inside_the_keys(lib, cuda, k, shift, inplace):
    """slot_src in the keys' own buffer or in another; buffers that are not aligned to 16
    bytes take single loads and stores instead of 16-byte ones."""
    from torchcor_b200._lib import check, ptr, stream_ptr
    from torchcor_b200.core.assemble import build_pattern
    el, n = _fans(k, [1, 5, 8, 16, 17, 32, 33, 64, 65, 200], np.random.default_rng(7 + k))
    E, h = len(el), build_pattern(el, n)
    d = torch.from_numpy(np.concatenate([np.zeros(shift, np.int32), el.reshape(-1)])).to(cuda)[shift:]
    work = torch.empty(2 * (n + 1), device=cuda, dtype=torch.int64)
    keys = torch.empty(k * k * E + shift, device=cuda, dtype=torch.int64)[shift:]
    iwork = torch.empty(2 * n + 1, device=cuda, dtype=torch.int32)
    nnz = C.c_int64()
    check(lib.tcb_pattern_device(ptr(d), E, k, n, ptr(work), ptr(keys), ptr(iwork), C.byref(nnz), stream_ptr()))
    i32 = dict(device=cuda, dtype=torch.int32)
    src = keys.view(torch.int32)[:k * k * E] if inplace else torch.empty(k * k * E, **i32)
    got = [torch.empty(n + 1, **i32), torch.empty(nnz.value, **i32), torch.empty(nnz.value + 1, **i32), src, torch.empty(n, **i32)]
    check(lib.tcb_pattern_device_emit(ptr(work), ptr(keys), E, k, n, *(ptr(t) for t in got), stream_ptr()))
    for name, t in zip(NAMES, got):
        assert np.array_equal(t.cpu().numpy(), h.host(name)), name


def test_far_columns_and_multi_block_scans(lib, cuda):
    """A strip of triangles over 4.3 million nodes, some joined to nodes millions of
    rows away: beyond the 22- and 23-bit column offsets of the register sorts."""
    n = 4_300_001
    i = np.arange(0, n - 2, 2, dtype=np.int64)
    strip = np.stack([i, i + 1, i + 2], 1)
    far = np.array([(0, n - 1, 5), (7, n // 2, n - 3), (n - 2, 1, n // 3)], dtype=np.int64)
    fan = np.array([(9, 20 + 2 * j, 4_200_000 + j) for j in range(45)], dtype=np.int64)
    _equal(np.concatenate([strip, far, fan]).astype(np.int32), n, cuda)


@pytest.mark.parametrize("n,widest", [(1, 1), (31, 5), (32, 7), (33, 40), (5000, 90), (300_000, 6)])
def test_sliced_ell_on_the_device(lib, cuda, n, widest):
    """Layout and packing against the host layout and a plain loop; rows of up to 90
    entries make slices beyond what a warp stages."""
    from torchcor_b200._lib import TCB_SLICE
    from torchcor_b200.core.assemble import Pattern, _sliced_ell
    rng = np.random.default_rng(n)
    length = rng.integers(1, widest + 1, size=n)
    rowptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
    nnz = int(rowptr[-1])
    col = rng.integers(0, n, size=nnz).astype(np.int32)
    vals = [rng.normal(size=nnz).astype(np.float32) for _ in range(3)]
    dev = [torch.from_numpy(a).to(cuda) for a in (rowptr, col, *vals)]
    pat = Pattern(n, 4, dev[0], dev[1], None, None, None, n_nonzero=nnz)
    ns, sp, scol, dcol, sell, flag = _sliced_ell(pat, dev[0], dev[1], dev[2:], cuda, torch.ones(1, device=cuda, dtype=torch.int32))
    assert flag
    want = np.empty(ns + 1, dtype=np.int64)
    ne = C.c_int64()
    assert lib.tcb_sell_layout(rowptr.ctypes.data, n, want.ctypes.data, C.byref(ne)) == 0
    assert np.array_equal(sp.cpu().numpy(), want)
    pc, pv = np.empty(ne.value, dtype=np.int32), [np.zeros(ne.value, dtype=np.float32) for _ in range(3)]
    for s in range(ns):
        w = int(want[s + 1] - want[s]) // TCB_SLICE
        for lane in range(TCB_SLICE):
            row = s * TCB_SLICE + lane
            at = want[s] + lane + TCB_SLICE * np.arange(w)
            pc[at] = row if row < n else 0
            if row < n:
                b, m = rowptr[row], length[row]
                pc[at[:m]] = col[b:b + m]
                for p, v in zip(pv, vals):
                    p[at[:m]] = v[b:b + m]
    assert np.array_equal(scol.cpu().numpy(), pc)
    for t, p in zip(sell, pv):
        assert np.array_equal(t.cpu().numpy(), p)


@pytest.mark.parametrize("nnz,shift", [(1, 0), (4, 0), (1023, 0), (4099, 0), (4099, 1)])
def test_system_values_in_vectors_and_one_by_one(lib, cuda, nnz, shift):
    """A, K / chi and K' at vector remainders and on arrays that are not aligned to 16 bytes,
    each float32 operation rounded by itself as in numpy: equal to the bit."""
    from torchcor_b200._lib import check, ptr, stream_ptr
    rng = np.random.default_rng(nnz)
    k, m = rng.normal(size=nnz).astype(np.float32), rng.uniform(0.1, 1, nnz).astype(np.float32)
    kd, md = (torch.from_numpy(np.concatenate([np.zeros(shift, np.float32), v])).to(cuda)[shift:] for v in (k, m))
    a, kr = (torch.zeros(nnz + shift, device=cuda)[shift:] for _ in range(2))
    d, diag = torch.zeros(1, device=cuda), torch.zeros(1, device=cuda, dtype=torch.int32)
    chi, cm, dt, theta = 140.0, 0.01, 0.01, 0.5
    split = torch.ones(1, device=cuda, dtype=torch.int32)
    check(lib.tcb_assemble_system(nnz, 1, 1, ptr(diag), ptr(kd), ptr(md), chi, cm, dt, theta, ptr(a), ptr(kr), ptr(d),
                                  ptr(split), stream_ptr()))
    f = np.float32
    kc, mc = k / f(chi), m * f(cm)
    want, wr = mc + kc * f(dt) * f(theta), kc * f((1 - theta) * dt)
    assert np.array_equal(kd.cpu().numpy(), kc) and np.array_equal(a.cpu().numpy(), want)
    assert np.array_equal(kr.cpu().numpy(), wr) and bool(split.item()) == bool(np.all(mc + wr == want))


@pytest.mark.parametrize("k", [3, 4])
def test_gather_of_the_last_contributions_below_2_31(lib, cuda, k):
    """Slots whose contributions end at 2^31 - 2, the most that the pattern build takes: sums of
    the last 5,000, in windows that an int32 counter would step over the end of."""
    from torchcor_b200._lib import check, ptr, stream_ptr
    rng = np.random.default_rng(k)
    total, tail, nnz, E = 2 ** 31 - 2, 5000, 300, 50
    cuts = np.sort(rng.choice(np.arange(1, tail), nnz - 1, replace=False))
    cuts = np.concatenate([[0], cuts, [tail]])
    src = rng.integers(0, k * k * E, tail).astype(np.int32)
    ke, mw = rng.normal(size=k * k * E).astype(np.float32), rng.normal(size=E).astype(np.float32)
    slot_ptr = torch.from_numpy((total - tail + cuts).astype(np.int32)).to(cuda)
    slot_src = torch.zeros(total, device=cuda, dtype=torch.int32)
    slot_src[total - tail:] = torch.from_numpy(src).to(cuda)
    d_ke, d_mw = torch.from_numpy(ke).to(cuda), torch.from_numpy(mw).to(cuda)
    out = torch.zeros((2, nnz), device=cuda, dtype=torch.float32)
    check(lib.tcb_assemble_gather(k, ptr(slot_ptr), ptr(slot_src), nnz, ptr(d_ke), ptr(d_mw), ptr(out[0]), ptr(out[1]),
                                  stream_ptr()))
    ab = src % (k * k)
    mass = mw[src // (k * k)] * np.where(ab // k == ab % k, np.float32(2), np.float32(1))
    want = np.zeros((2, nnz), dtype=np.float32)
    for s in range(nnz):
        for j, v in enumerate((ke[src], mass)):
            # float32 sums one by one, in order
            want[j, s] = np.add.accumulate(v[cuts[s]: cuts[s + 1]], dtype=np.float32)[-1]
    assert np.array_equal(out.cpu().numpy(), want)
    del slot_src
    torch.cuda.empty_cache()


def test_element_matrices_divide_by_the_determinant(lib, cuda):
    """Tetrahedra on the axes with edges 1, 2, m: the gradient along the first is (2 m) / (2 m) = 1 and
    K[1][1] = volume * sigma is half way between two float32 values, so that it rounds to the even one
    only if the quotient is rounded once.  The determinants are those for which the product with
    the reciprocal is below 1."""
    from torchcor_b200._lib import check, ptr, stream_ptr
    dets, sigma = [], []
    for det in range(12, 60000, 12):                      # volume det / 6, m = det / 2
        if float(det) * (1.0 / det) >= 1.0:
            continue
        for j in range(1, 256):
            s = 1.0 + j * 2.0 ** -23
            v = det / 6 * s                               # exact: 13 and 24 bits
            below = v * (1 - 2.0 ** -53)
            if np.float32(v) > np.float32(below):
                dets.append(det)
                sigma.append(s)
                break
    E = len(dets)
    assert E >= 20
    nodes = np.zeros((E, 4, 3), dtype=np.float32)
    nodes[:, 1, 0], nodes[:, 2, 1], nodes[:, 3, 2] = 1, 2, np.array(dets) / 2
    elems = np.arange(4 * E, dtype=np.int32).reshape(E, 4)
    fib = np.tile(np.array([1, 0, 0], dtype=np.float32), (E, 1))
    d = [torch.from_numpy(a).to(cuda) for a in (nodes.reshape(-1, 3), elems, np.array(sigma, dtype=np.float32), fib)]
    ke, mw = torch.empty((E, 16), device=cuda), torch.empty(E, device=cuda)
    check(lib.tcb_assemble_local(4, ptr(d[0]), ptr(d[1]), E, ptr(d[2]), ptr(d[2]), ptr(d[3]), ptr(ke), ptr(mw), stream_ptr()))
    want = (np.array(dets) / 6 * np.array(sigma)).astype(np.float32)
    assert np.array_equal(ke[:, 5].cpu().numpy(), want)


def test_nodes_in_no_element_on_the_device(lib, cuda):
    """The device pattern takes nodes that no element has: empty rows, -1 for the diagonal slot, 0 for
    the preconditioner; the other nodes' values are those of the mesh without them."""
    from torchcor_b200 import meshgen
    from torchcor_b200.core.assemble import assemble_system, build_pattern_device
    nodes, elems = meshgen.cube(5, 0.25)
    n, gaps = len(nodes), [0, 40, 41, 216]
    keep = np.setdiff1d(np.arange(n + len(gaps)), gaps)
    wide = np.zeros((n + len(gaps), 3), dtype=np.float32)
    wide[keep] = nodes
    spread = keep[elems].astype(np.int32)
    pat = build_pattern_device(torch.from_numpy(spread).to(cuda), len(wide))
    assert (pat.host("diag")[gaps] == -1).all() and (np.diff(pat.host("rowptr"))[gaps] == 0).all()
    assert (pat.host("col")[pat.host("diag")[keep]] == keep).all()
    fib = torch.tensor([[1.0, 0, 0]], device=cuda).repeat(len(elems), 1).contiguous()
    s = torch.full((len(elems),), 0.3, device=cuda)
    def system(x, el):
        return assemble_system(torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).to(cuda),
                               torch.from_numpy(np.ascontiguousarray(el, dtype=np.int32)).to(cuda), s, s, fib, 0.01)
    a, b = system(wide, spread), system(nodes, elems)
    assert (a.d_inv[gaps] == 0).all()
    assert torch.equal(a.d_inv[torch.from_numpy(keep).to(cuda)], b.d_inv[:n])
    assert torch.equal(a.a_val, b.a_val) and torch.equal(a.k_val, b.k_val)
