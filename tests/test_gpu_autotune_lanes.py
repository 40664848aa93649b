"""The autotuner leaves pr_tile_u alone where no plan follows it, and searches it where
one does."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,follows", [(10, False), (15, False), (19, True)])
def test_lanes_are_searched_where_they_matter(scale, follows):
    import olive_b200 as ob
    with ob.Graph.rmat(scale, 16, seed=2) as g:
        before = g.pagerank(max_it=4, tol=0.0)
        g.tune(pr_tile_u=32)
        assert (g.pagerank(max_it=4, tol=0.0).tobytes() == before.tobytes()) == (not follows)
        assert (g.autotune(reps=1)["pr_tile_u"] in (4, 8, 16)) == follows
