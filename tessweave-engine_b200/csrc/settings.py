"""Switches of the environment, read anew at every use.

``os.environ.get`` of a name that is not set raises and catches an exception inside, one microsecond each time; a step that is
launched kernel by kernel asks for more than a hundred, mostly unset, which was a tenth of its host time.  The mapping keeps its
entries as a dictionary of bytes on POSIX; where it does not, or where another mapping stands in its place, that is asked itself.
"""
from __future__ import annotations

import os

_environ = os.environ
_entries = getattr(_environ, "_data", None) if os.name == "posix" else None


def setting(name: str, default: str | None = None) -> str | None:
    """``os.environ.get(name, default)``."""
    if _entries is None or os.environ is not _environ:
        return os.environ.get(name, default)
    raw = _entries.get(name.encode())
    return default if raw is None else os.fsdecode(raw)
