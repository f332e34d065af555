"""A test that needs hilbert's compiled code skips where it is not built."""
import pytest

import conftest
import oracle.doci
import oracle.maps


@pytest.mark.parametrize("mod", [oracle.maps, oracle.doci])
def test_missing_reference_is_a_skip(mod, monkeypatch, request):
    monkeypatch.setattr(mod, "ref_available", lambda: False)
    load = mod._ref_lib if mod is oracle.maps else (lambda: mod._lib("ref"))
    monkeypatch.setattr(mod, "_rlib", None, raising=False)
    monkeypatch.setattr(mod, "_libs", {}, raising=False)
    wrapper = conftest.pytest_runtest_call(request.node)
    next(wrapper)
    with pytest.raises(pytest.skip.Exception):
        try:
            load()
        except FileNotFoundError as e:
            wrapper.throw(e)
