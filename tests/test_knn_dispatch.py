"""Which kernel a neighbour search takes, asked of the library's own rule (no GPU)."""
import pytest

from nngpr_b200 import _lib

TC, SIMT, GENERIC, DIRECT = range(4)


@pytest.fixture(autouse=True)
def automatic(monkeypatch):
    monkeypatch.delenv('NNGP_KNN_KERNEL', raising=False)


def path(n_ref, n_query, d, m=32, cut=None, f64=False):
    return _lib.lib().nngp_knn_path(n_ref, n_query, d, m, int(cut is not None), cut or 0, int(f64))


@pytest.mark.parametrize('d', [1, 3, 6, 8, 10, 12, 14, 16, 18, 20])
def test_a_set_over_itself_is_direct_up_to_one_size(d):
    """One line for prefix searches: direct below it, tensor-core above it, none in between."""
    kinds = [path(n, n, d, cut=0) for n in (500, 2000, 8191, 8192, 12000, 14000, 16383, 16384)]
    assert kinds == [DIRECT] * 8
    assert [path(n, n, d, cut=0) for n in (16385, 20000, 65536, 434874)] == [TC] * 4


def test_a_set_of_24_features_turns_where_the_pairs_cost_more():
    kinds = [path(n, n, 24, cut=0) for n in range(1000, 30000, 250)]
    first = kinds.index(TC)
    assert set(kinds[:first]) == {DIRECT} and set(kinds[first:]) == {TC}
    assert 12000 <= 1000 + 250 * first <= 16384


@pytest.mark.parametrize('d', [3, 8, 12, 16, 18])
def test_equal_counts_are_no_prefix_search(d):
    """Queries that happen to be as many as the refs cost all pairs; a neighbouring count takes the same path."""
    near = [path(n, 16384, d) for n in (16000, 16383, 16384, 16385, 17000)]
    assert len(set(near)) == 1
    assert len({path(16384, nq, d) for nq in (16384, 16385, 17000)}) == 1


@pytest.mark.parametrize('d', [3, 8, 16, 24])
@pytest.mark.parametrize('cut', [None, 0])
def test_more_queries_never_turn_a_search_back_to_direct(d, cut):
    for n_ref in (500, 16384, 50000, 434874):
        kinds = [path(n_ref, nq, d, cut=cut) for nq in (1, 100, 1000, 4000, 9000, 16383, 16384, 16385, 30000, 100000)]
        first = kinds.index(TC) if TC in kinds else len(kinds)
        assert set(kinds[:first]) <= {DIRECT} and set(kinds[first:]) <= {TC}


@pytest.mark.parametrize('d,m,below,above', [(3, 48, 45000, 60000), (8, 64, 45000, 60000), (16, 48, 20000, 25000),
                                             (26, 32, 11000, 13000), (32, 32, 9500, 11000)])
def test_against_the_simt_screen_queries_count_by_their_refs(d, m, below, above):
    """The same line for any number of refs; a set over itself has half the pairs, so twice the points."""
    for n_ref in (20000, 100000, 434874):
        assert path(n_ref, below, d, m) == DIRECT and path(n_ref, above, d, m) == SIMT
    assert path(2 * below, 2 * below, d, m, cut=0) == DIRECT and path(2 * above, 2 * above, d, m, cut=0) == SIMT


def test_fp64_and_other_shapes():
    assert path(434874, 434874, 3, cut=0, f64=True) == DIRECT and path(1000, 10, 3, 200, f64=True) == GENERIC
    assert path(100000, 50, 40) == DIRECT and path(100000, 50, 3, 200) == GENERIC
    assert path(10, 0, 3) == -1


@pytest.mark.parametrize('f64', [False, True])
@pytest.mark.parametrize('n_ref,n_query,d,m', [(16384, 16384, 8, 32), (16384, 16384, 12, 32), (20000, 16384, 16, 32),
                                               (100000, 9000, 3, 32), (434874, 1000, 3, 32), (50000, 30000, 8, 48)])
def test_the_workspace_serves_the_search_with_and_without_a_cut(monkeypatch, f64, n_ref, n_query, d, m):
    """The size functions are not told of a cut: the size covers the kernels that either search takes."""
    L = _lib.lib()
    size = L.nngp_knn_workspace_size_f64 if f64 else L.nngp_knn_workspace_size_f32
    auto = size(n_ref, n_query, d, m)
    for cut in (None, 0, -5, n_ref // 2):
        k = path(n_ref, n_query, d, m, cut, f64)
        monkeypatch.setenv('NNGP_KNN_KERNEL', ('tc', 'simt', 'generic', 'direct')[k])
        assert auto >= size(n_ref, n_query, d, m)
        monkeypatch.delenv('NNGP_KNN_KERNEL')


def test_the_bench_counts_the_launches_of_the_search_it_runs():
    import bench
    for n, d in ((2000, 3), (8192, 16), (16384, 16)):
        assert path(n, n, d, cut=0) == DIRECT and bench.our_launches_per_step(n, d, 32) == 4
    assert bench.our_launches_per_step(16385, 16, 32) > 4
