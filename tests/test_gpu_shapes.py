"""Volumes of extreme shape on the GPU against the oracle: thin along one axis and long
along another, down to the smallest accepted size (4 voxels per axis, a 2-voxel
interior), registered as one cohort with either staging and compared pair by pair with
the oracle bit for bit.  An empty cohort and a volume below the minimum are refused with
a status, and the handle registers correctly afterwards."""
import numpy as np
import pytest

from fastreg_gb300 import FastReg, Params, _native as N
from oracle import oracle as O
from tests.helpers import assert_bitexact, images

pytestmark = pytest.mark.gpu

# (X, Y, Z): one voxel-pitch chunk wide in x (4), rows of one or two tiles, 70 slices, a
# row pitch padded from 97 to 100, and the minimum cube
SHAPES = [(4, 45, 5), (70, 4, 6), (5, 6, 70), (97, 5, 4), (4, 4, 4)]


def _to(dev, a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def _check_pair(solver, P, p, buf, psi, what):
    if solver == "reference":
        o = O.ref_register(P, p["T"], p["labT"], p["S"], p["labS"])
        assert_bitexact(psi, o["psi"], f"{what} psi")
        assert_bitexact(buf[0].cpu().numpy(), o["out_T"], f"{what} T o psi_inv")
        assert_bitexact(buf[1].cpu().numpy(), o["out_labT"], f"{what} labels T o psi_inv")
        assert_bitexact(buf[2].cpu().numpy(), o["out_S"], f"{what} S o psi")
        assert_bitexact(buf[3].cpu().numpy(), o["out_labS"], f"{what} labels S o psi")
    else:
        o = O.sob_register(P, p["T"], p["S"])
        assert_bitexact(psi, o["phi"], f"{what} phi")
        assert_bitexact(buf[2].cpu().numpy(), O.warp(o["phi"], p["S"]), f"{what} S o phi")
        assert_bitexact(buf[3].cpu().numpy(), O.warp_nearest_label(o["phi"], p["labS"]), f"{what} labels")


@pytest.mark.parametrize("staging", [1, 2])
@pytest.mark.parametrize("solver", ["reference", "sobolev"])
def test_extreme_shapes_as_one_cohort(cuda, solver, staging):
    kw = dict(no_labels=4, max_iter=15, alpha=0.02, solver=solver, step=0.5, damping=0.9, staging=staging)
    pairs_np = [images(d, 1700 + k) for k, d in enumerate(SHAPES)]
    fr = FastReg(Params(volume_dims=SHAPES[0], **kw))
    bufs = [tuple(_to(cuda, p[k]) for k in ("T", "labT", "S", "labS")) for p in pairs_np]
    fr.register_batch(bufs)
    for k, (d, p) in enumerate(zip(SHAPES, pairs_np)):
        psi = fr.get_field(N.FR_FIELD_PSI, pair=k).cpu().numpy()
        _check_pair(solver, Params(volume_dims=d, **kw), p, bufs[k], psi, f"pair {k} {d}")
        assert fr.stats(pair=k).iterations == 15
    fr.close()


def test_empty_and_undersized_cohorts_are_refused(cuda):
    from fastreg_gb300._native import FastRegError
    kw = dict(no_labels=4, max_iter=10, alpha=0.02)
    fr = FastReg(Params(volume_dims=(12, 10, 9), **kw))
    with pytest.raises(FastRegError, match="at least one pair"):
        fr.register_batch([])
    small = images((3, 10, 10), 1800)
    with pytest.raises(FastRegError, match="< 4"):
        fr.register_batch([tuple(_to(cuda, small[k]) for k in ("T", "labT", "S", "labS"))])
    # the handle still works
    p = images((12, 10, 9), 1801)
    buf = tuple(_to(cuda, p[k]) for k in ("T", "labT", "S", "labS"))
    fr(*buf)
    _check_pair("reference", Params(volume_dims=(12, 10, 9), **kw), p, buf,
                fr.get_field(N.FR_FIELD_PSI).cpu().numpy(), "after the refusals")
    fr.close()


@pytest.mark.parametrize("dims", [(1, 1, 1), (31, 1, 1), (1, 63, 1), (4, 4, 4), (5, 13, 1), (3, 1, 43), (43, 3, 1), (9, 7, 61)])
def test_field_operations_at_remainders(cuda, dims):
    """fr_warp and fr_interpolate_field where the last item of a warp's 64 voxels is partly or
    nearly empty, on buffers that are only element-aligned: the oracle's bits."""
    import torch
    from fastreg_gb300 import interpolate_field, warp
    X, Y, Z = dims
    r = np.random.Generator(np.random.PCG64(17))
    img, lab = r.normal(0, 1, (Z, Y, X)).astype(np.float32), r.integers(0, 9, (Z, Y, X)).astype(np.int16)
    field = r.normal(0, 1, (3, Z, Y, X)).astype(np.float32)
    pos = np.stack([r.uniform(-1, n, (Z, Y, X)) for n in dims]).astype(np.float32)

    def shifted(a):  # one element past an allocation's start
        t = torch.empty(a.size + 1, dtype=torch.from_numpy(a).dtype, device=cuda)[1:].view(a.shape)
        t.copy_(torch.from_numpy(a))
        return t

    for to in (lambda a: _to(cuda, a), shifted):
        out, out_lab = to(np.zeros_like(img)), to(np.zeros_like(lab))
        warp(to(pos), to(img), to(lab), out=out, out_lab=out_lab)
        o_img, o_lab = O.warp(pos, img, lab)
        assert_bitexact(out.cpu().numpy(), o_img, f"warp {dims}")
        assert_bitexact(out_lab.cpu().numpy(), o_lab, f"warp labels {dims}")
        assert_bitexact(warp(to(pos), to(img)).cpu().numpy(), o_img, f"warp without labels {dims}")
        assert_bitexact(interpolate_field(to(field), to(pos), out=to(np.zeros_like(field))).cpu().numpy(),
                        O.interpolate_field(field, pos), f"field {dims}")


@pytest.mark.parametrize("dims", [(2, 2, 2), (33, 9, 2), (31, 8, 40), (70, 17, 33)])
def test_warp_adjoint_over_sizes(cuda, dims):
    """fr_warp_adjoint at tile edges, single-slice columns and columns longer than a tile, maps that
    keep cells stacked (a uniform shift) and that do not (noise), outside positions and a NaN;
    both outputs, and each alone.  A voxel of img_bar sums a few dozen FP32 terms in any
    order, a component of pos_bar about ten: 1e-5 of the largest value, as in the test of one size."""
    import ctypes as C
    import torch
    lib = N.load()
    X, Y, Z = dims
    r = np.random.Generator(np.random.PCG64(23))
    img, wbar = (r.normal(0, 1, (Z, Y, X)).astype(np.float32) for _ in range(2))
    grid = np.stack(np.meshgrid(np.arange(Z), np.arange(Y), np.arange(X), indexing="ij")[::-1]).astype(np.float32)
    for pos in (grid + np.float32(0.3), grid + r.uniform(-2.5, 2.5, grid.shape).astype(np.float32)):
        pos[:, 0, 0, 0] = np.nan
        pb64, ib64 = O.warp_adjoint(pos, img, wbar)
        a = [_to(cuda, v) for v in (pos, img, wbar)]
        for want_pos, want_img in ((1, 1), (1, 0), (0, 1)):
            pb, ib = torch.empty_like(a[0]), torch.empty_like(a[1])
            assert lib.fr_warp_adjoint(*(v.data_ptr() for v in a), (C.c_int * 3)(*dims), pb.data_ptr() if want_pos else None,
                                       ib.data_ptr() if want_img else None, None) == N.FR_OK
            if want_pos:
                assert np.abs(pb.cpu().numpy() - pb64).max() <= 1e-5 * max(1.0, np.abs(pb64).max())
            if want_img:
                assert np.abs(ib.cpu().numpy() - ib64).max() <= 1e-5 * max(1.0, np.abs(ib64).max())


@pytest.mark.parametrize("dims", [(7, 9, 3001), (1, 3, 70001), (24, 24, 301), (601, 17, 40), (31, 33, 700)])
def test_field_sampling_columns_of_narrow_volumes(cuda, dims):
    """fr_interpolate_field where a block's columns run on over several slices and their last layer is
    shorter than the others: the oracle's bits."""
    from fastreg_gb300 import interpolate_field
    X, Y, Z = dims
    r = np.random.Generator(np.random.PCG64(19))
    field = r.normal(0, 1, (3, Z, Y, X)).astype(np.float32)
    grid = np.stack(np.meshgrid(np.arange(Z), np.arange(Y), np.arange(X), indexing="ij")[::-1]).astype(np.float32)
    for pos in (grid + np.float32(0.25), grid + r.uniform(-2, 2, grid.shape).astype(np.float32)):
        assert_bitexact(interpolate_field(_to(cuda, field), _to(cuda, pos)).cpu().numpy(),
                        O.interpolate_field(field, pos), f"field {dims}")


@pytest.mark.parametrize("dims", [(5, 300, 301), (16, 31, 20), (33, 33, 100), (3, 130, 9), (4, 4, 20001), (2, 3, 5000),
                                  (15, 9, 700)])
def test_warp_adjoint_of_narrow_volumes(cuda, dims):
    """fr_warp_adjoint where its blocks are less than 32 columns wide (16 x 16, 8 x 32, 4 x 64) or hold
    several layers of columns, the last of them shorter or empty: as test_warp_adjoint_over_sizes."""
    test_warp_adjoint_over_sizes(cuda, dims)
