from ._lib import release_scratch  # noqa: F401
