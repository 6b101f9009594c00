"""First-order batches whose chunks change to the pair flux, with just fewer and just more chunks than its form for
large grids takes, and few: every tube ends in the bits of the same tube run alone, whose run is resident."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,cfl", [("mixed_f64", 0.25), ("mixed_kahan", 0.2)])
@pytest.mark.parametrize("chunks_per_sm", [1.2, 7.9, 8.1])
def test_tubes_of_a_batch_match_themselves_alone(shll, chunks_per_sm, prec, cfl):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 5000                                   # 11 chunks
    count = int(chunks_per_sm * sms / 11)
    items = [shll.params(1, 1, nx=n + t % 3, precision=prec, cfl=cfl, fold_steps=64, n_steps=100 + 16 * (t % 2),
                         ic_rho_l=2.0 + 40.0 * (t % 5), ic_T_l=1.2, ic_x_d=0.3 + 0.05 * (t % 7)) for t in range(count)]
    b = shll.Batch(items)
    b.run()
    for t in list(range(0, 8)) + [count // 2, count - 1]:
        c = shll.Context(items[t])
        c.init_state()
        c.run()
        assert np.array_equal(b.primitives(t), c.primitives()), t
        c.close()
    b.close()
