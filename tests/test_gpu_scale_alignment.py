"""Scale buffers at any byte address: off a 4-byte boundary they are stored byte by byte, the bytes of an aligned buffer, and none beside them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# few rows: narrow ones, one group a thread, two (their groups shared by CTAs, and not); many rows: one and several warps per set; the widest rows
@pytest.mark.parametrize("rows, k, ke, mode, forms", [
    (9, 64, 16, 16, "plain given own weight"), (33, 1040, 48, 16, "plain given own weight"), (16, 4096, 128, 16, "plain given own rms"),
    (889, 4096, 0, 16, "plain given own"), (16, 14336, 64, 16, "plain given own weight"), (300, 9216, 96, 32, "plain given"), (2001, 1024, 64, 16, "rms"),
    (4001, 512, 512, 16, "plain own"), (2001, 4112, 80, 16, "plain given own weight"), (2001, 4096, 128, 16, "rms"), (1801, 14336, 128, 32, "plain own"),
    (40, 18944, 64, 32, "plain")])
def test_any_address(rows, k, ke, mode, forms):
    from arcquant_b200 import _lib, ops

    lib, st = _lib.load(), ops._stream()
    x = torch.randn(rows, k, device="cuda").bfloat16()
    idx, gain = torch.randperm(k).to(torch.int16).cuda(), torch.randn(k, device="cuda").bfloat16()
    one, scale, scratch = torch.full((), 0.37, device="cuda"), torch.empty(1, device="cuda"), torch.empty(_lib.SCALE_SCRATCH, device="cuda")
    n = ops.sf_bytes(rows, k + ke)
    for form in forms.split():
        def call(sf):
            q = torch.zeros(rows, (k + ke) // 2, dtype=torch.uint8, device="cuda")
            a, z = (x.data_ptr(), idx.data_ptr()), (q.data_ptr(), sf.data_ptr())
            rc = {"plain": lambda: lib.arcq_reorder_quantize_x(*a, rows, k, ke, mode, *z, st),
                  "weight": lambda: lib.arcq_reorder_quantize_w(*a, rows, k, ke, mode, *z, st),
                  "given": lambda: lib.arcq_reorder_quantize_x_scaled(a[0], one.data_ptr(), a[1], rows, k, ke, mode, *z, st),
                  "own": lambda: lib.arcq_quantize_tensor_scale(a[0], None, 0, a[1], rows, k, ke, mode, *z, scale.data_ptr(), scratch.data_ptr(), st),
                  "rms": lambda: lib.arcq_rmsnorm_quantize_x(a[0], gain.data_ptr(), 1e-5, a[1], rows, k, ke, *z, st)}[form]()
            assert rc == 0, (form, rc)
            return q
        want_sf = torch.full((n,), 0xa5, dtype=torch.uint8, device="cuda")
        want = call(want_sf)
        for off in (1, 2, 3, 4):
            room = torch.full((n + 16,), 0xa5, dtype=torch.uint8, device="cuda")
            assert torch.equal(call(room[off:off + n]), want)
            assert torch.equal(room[off:off + n], want_sf), (form, off)
            assert bool((room[:off] == 0xa5).all()) and bool((room[off + n:] == 0xa5).all())


@pytest.mark.parametrize("k, rows", [(256, 512), (2048, 512), (2048, 6400), (14336, 512), (14336, 2304)])      # narrow rows, few rows and many
def test_any_address_of_grouped_rows(k, rows):
    from arcquant_b200 import _lib, ops

    lib, st, e, ke = _lib.load(), ops._stream(), 2, 64
    x = torch.randn(rows, k, device="cuda").bfloat16()
    idx = torch.stack([torch.randperm(k) for _ in range(e)]).to(torch.int16).cuda()
    half = rows // 512 * 256
    groups, amax, scale = torch.tensor([0, half, half - 3, rows - half], dtype=torch.int32, device="cuda"), torch.full((e,), 5.0, device="cuda"), torch.empty(e, device="cuda")
    n = ops.sf_bytes(rows, k + ke)

    def call(sf):
        q = torch.zeros(rows, (k + ke) // 2, dtype=torch.uint8, device="cuda")
        assert lib.arcq_quantize_x_grouped_amax(x.data_ptr(), None, amax.data_ptr(), idx.data_ptr(), groups.data_ptr(), e, rows, k, ke, 16, q.data_ptr(),
                                                sf.data_ptr(), scale.data_ptr(), st) == 0
        return q

    want_sf = torch.full((n,), 0xa5, dtype=torch.uint8, device="cuda")
    want = call(want_sf)
    for off in (1, 2, 3):
        room = torch.full((n + 16,), 0xa5, dtype=torch.uint8, device="cuda")
        assert torch.equal(call(room[off:off + n]), want) and torch.equal(room[off:off + n], want_sf)
        assert bool((room[:off] == 0xa5).all()) and bool((room[off + n:] == 0xa5).all())
