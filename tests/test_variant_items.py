"""What lgm_variant_items reports of each variant (no GPU needed)."""
import langmuir_b200 as L


def test_items_per_variant():
    vs = L.Coulomb.variants()
    default = vs.pop()
    # r^2 from the tensor cores: items chosen per call
    assert default["culled"] and default["run"] == 16 and not default["warp_specialised"]
    assert default["chunks_per_item"] == 0 and default["stages"] == 0
    for v in vs:
        assert (v["chunks_per_item"] > 0) == v["culled"]
        assert (v["stages"] > 0) == v["warp_specialised"]
