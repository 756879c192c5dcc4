"""ROPE from a table of angles and the K/V store: bit-identical to b200_rope_store, which works the angles out itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# heads that do not fill the last CTA, every head size, rotated dims short of the head, packed and stacked rows
@pytest.mark.parametrize("T,D,H,Hkv,n_dims,stacked", [(1, 64, 32, 8, 64, True), (3, 128, 4, 2, 128, False), (2, 256, 3, 1, 128, True), (64, 128, 32, 8, 128, True), (5, 64, 7, 1, 32, False)])
def test_rope_store_angles(T, D, H, Hkv, n_dims, stacked):
    from cactus_b200._lib import check, lib
    L, cells = lib(), 80
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(T + D)
    qd, kvd = H * D, Hkv * D
    if stacked:
        qkv = torch.randn((T, qd + 2 * kvd), device="cuda", generator=g)
        parts = lambda x: (x[:, :qd], x[:, qd:qd + kvd], x[:, qd + kvd:])  # noqa: E731
        a, b = parts(qkv.clone()), parts(qkv.clone())
    else:
        rows = [torch.randn((T, n), device="cuda", generator=g) for n in (qd, kvd, kvd)]
        a, b = [r.clone() for r in rows], [r.clone() for r in rows]
    pos = torch.randint(0, 5000, (T,), device="cuda", generator=g, dtype=torch.int32)
    slots = torch.randperm(cells, device="cuda", generator=g)[:T].to(torch.int32)
    caches = [torch.zeros((cells, kvd), dtype=torch.float16, device="cuda") for _ in range(4)]
    rope = (n_dims, pos.data_ptr(), None, 500000.0, 0.5, 1.1)
    shape = lambda x: (x[0].data_ptr(), D * 4, x[0].stride(0) * 4, x[1].data_ptr(), D * 4, x[1].stride(0) * 4, x[2].data_ptr(), x[2].stride(0) * 4, D, H, Hkv, T)  # noqa: E731
    check(L.b200_rope_store(*shape(a), *rope, slots.data_ptr(), caches[0].data_ptr(), kvd * 2, caches[1].data_ptr(), kvd * 2, st))
    angles = torch.empty((T, n_dims), device="cuda")
    check(L.b200_rope_angles(angles.data_ptr(), T, *rope, st))
    check(L.b200_rope_store_angles(*shape(b), n_dims, angles.data_ptr(), slots.data_ptr(), caches[2].data_ptr(), kvd * 2, caches[3].data_ptr(), kvd * 2, st))
    torch.cuda.synchronize()
    for x, y in zip((*a, *caches[:2]), (*b, *caches[2:])):
        assert torch.equal(x, y)


@pytest.mark.parametrize("T", [1, 300])
def test_ubatch_begin(T):
    from cactus_b200._lib import check, lib
    L, cells, n_dims = lib(), 512, 128
    st = torch.cuda.current_stream().cuda_stream
    slots = torch.randperm(cells, device="cuda")[:T].to(torch.int32)
    pos, seq = (torch.randint(0, 5000, (T,), device="cuda", dtype=torch.int32) for _ in range(2))
    cell = [torch.full((cells,), -1, dtype=torch.int32, device="cuda") for _ in range(4)]
    angles = [torch.empty((T, n_dims), device="cuda") for _ in range(2)]
    check(L.b200_scatter_i32(cell[0].data_ptr(), slots.data_ptr(), pos.data_ptr(), T, st))
    check(L.b200_scatter_i32(cell[1].data_ptr(), slots.data_ptr(), seq.data_ptr(), T, st))
    check(L.b200_rope_angles(angles[0].data_ptr(), T, n_dims, pos.data_ptr(), None, 500000.0, 1.0, 1.0, st))
    check(L.b200_ubatch_begin(cell[2].data_ptr(), cell[3].data_ptr(), slots.data_ptr(), pos.data_ptr(), seq.data_ptr(), T, angles[1].data_ptr(), n_dims, None,
                              500000.0, 1.0, 1.0, st))
    torch.cuda.synchronize()
    assert torch.equal(cell[0], cell[2]) and torch.equal(cell[1], cell[3]) and torch.equal(*angles)
