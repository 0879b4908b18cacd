"""The tests run on a tuning cache of their own: the machine's one would change which variants and cells they test."""
import os


def test_the_tests_do_not_read_the_machines_cache():
    path = os.environ.get("SPH_TUNE_CACHE", "")
    assert path and not path.startswith(os.path.join(os.path.expanduser("~"), ".cache"))
