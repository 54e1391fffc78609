"""Set-ups on two host threads at once, a handle each, with bottoms that need
different amounts of shared memory: what one thread asks of a kernel must not
take anything from the other's launch."""
import threading

import numpy as np
import pytest

from oracle import problem as P

pytestmark = pytest.mark.gpu


# systems of order 102 and 15, bottoms of 3136 columns and of 4 that are 76 nodes high
@pytest.mark.parametrize("first,second", [((8, 8, 66), (8, 8, 8)), ((112, 112, 2), (4, 4, 150))])
def test_bottoms_of_two_sizes(first, second):
    import stzpp_gb300 as sg
    start, failed = threading.Barrier(2), []

    def work(dims):
        m, n, o = dims
        per = (True, True, o == 2)
        st, fix = sg.elastic_stencil(1.0, 2.0, *P.grid_spacing(m, n, o, per, h=1.0 / 8))
        st = np.array(st).reshape(27, 3, 3)
        st[13] += np.diag(np.diag(st[13]))
        b = np.random.default_rng(2).standard_normal((m * n * o, 3))
        try:
            with sg.Multigrid(dims, per, precision="fp64", max_coarse=m * n * o // 3, bottom="direct") as mg:
                want = None
                start.wait()
                for _ in range(150):
                    mg.setup_matrices(stencil=st.reshape(27, 9), fix=fix)
                    mg.setup_fields(r=b)
                    mg.v_cycle()
                    x = mg.get_x()
                    if want is None:
                        want = x
                    if not np.array_equal(x, want):
                        failed.append((dims, "another solution"))
                        return
        except Exception as e:   # a failed launch comes as a status
            failed.append((dims, str(e)))
            start.abort()

    threads = [threading.Thread(target=work, args=(d,)) for d in (first, second)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
