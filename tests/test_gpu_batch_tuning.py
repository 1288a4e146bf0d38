"""The batch autotuner's cache: a choice measured on one side of the resident
loop's size is not taken on the other, where staged tiles are another kernel."""
import pytest

from multigpuegtsmoothing_b200 import datagen

pytestmark = pytest.mark.gpu


def test_cache_knows_the_loop(capi):
    # one size bucket (2^17), k that no other test uses; the resident loop ends at 151,552 points
    tuned = []
    for n in (80000, 50000, 55000, 78000):
        b = capi.Batch([(datagen.sphere_cloud(n, 0.01, n), 37), (datagen.sphere_cloud(n, 0.01, n + 1), 37)])
        b.run(3)
        tuned.append(b.timings()["tune_ms"] > 0)
        b.close()
    assert tuned == [True, True, False, False]
