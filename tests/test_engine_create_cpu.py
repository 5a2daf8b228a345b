"""An engine configuration that is refused allocates nothing: the refusal comes
before the first device call, so it is the same without a GPU."""
import pytest

from sycldb_gb300 import capi
from sycldb_gb300.engine import Engine


@pytest.mark.parametrize("cfg", [{"plan_cache": -1}, {"join_tables": 3}, {"join_tables": -1}, {"segment_rows": 100}])
def test_refused_configurations(cfg):
    with pytest.raises(capi.SdbError) as e:
        Engine(**cfg)
    assert e.value.status == capi.SDB_ERR_INVALID
