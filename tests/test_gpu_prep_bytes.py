"""csu_prep_bytes, which the server's admission adds up, covers what a pack of the solves allocates: cells padded to whole
blocks and the maps from cells to solves included."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("viscous,scheme", [(None, "DPLUR"), ("sst", "DPLUR"), ("sa", "LUSGS"), (None, "RK")])
def test_pack_fits_in_the_sum(native, viscous, scheme):
    import csu_b200
    from csu_b200 import meshgen
    preps = []
    for n in (260, 300, 520, 777, 1030):
        su2, inp = meshgen.bump(ncells=n, mach=0.5, viscous=viscous, re=2e6 if viscous else None, order=1, n_linear=4,
                                cfl=1.0, scheme=scheme, flux="AUSM")
        preps.append(csu_b200.Prep(csu_b200.Case.from_text(inp, su2)))
    native.csu_pack_arena_release()  # a fresh arena: a quarter more than the pack needs
    pack = csu_b200.Pack(preps)
    need = pack.stats()["device_bytes"] / 1.25 - 256
    history = 1024 * (preps[0].nvar + 4) * 8
    assert sum(p.bytes - history for p in preps) >= need
    pack.close()
    native.csu_pack_arena_release()
