"""Pages taken many at a time: the ones that single calls would give, and a table whose array follows."""
import pytest

from infinilm_b200.cache.manager import OutOfPages, PagePool, PageTable


@pytest.mark.parametrize("n", [0, 1, 5, 8])
def test_taken_pages_are_those_of_single_calls(n):
    one, many = PagePool(8), PagePool(8)
    for p in (one, many):
        a, b = p.alloc(), p.alloc()
        p.free(b), p.free(a)
    assert many.take(n) == [one.alloc() for _ in range(n)]
    assert many.held() == one.held() and many.n_free == one.n_free
    with pytest.raises(OutOfPages):
        many.take(9 - n)
    assert many.held() == one.held() and many.n_free == one.n_free


@pytest.mark.parametrize("sub", [1, 4])
@pytest.mark.parametrize("k", [0, 1, 15, 16, 17, 200])
def test_a_table_extended_while_its_array_is_behind(sub, k):
    t = PageTable(sub=sub)
    t.extend(range(k))
    t += list(range(40))                          # (marks the array as behind, and outgrows it)
    t.extend([3, -1, 7] * 20)
    t.append(9)
    assert t.array().tolist() == [(-1 if p < 0 else p * sub + j) for p in t for j in range(sub)]
    t.extend([5, -1])
    t.append(1)
    assert t.array().tolist() == [(-1 if p < 0 else p * sub + j) for p in t for j in range(sub)]
