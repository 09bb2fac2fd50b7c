"""Device memory that Python objects keep for their next use and can do without: it goes back when the library is asked for its idle memory
(`api.mem_trim`) and before an array's allocation fails."""
from __future__ import annotations

import weakref

_holders: "weakref.WeakSet" = weakref.WeakSet()


def register(holder) -> None:
    """`holder.give_back()` frees what it keeps and says whether that was anything; work in flight keeps what it uses (freeing waits)."""
    _holders.add(holder)


def give_back() -> bool:
    return any([h.give_back() for h in list(_holders)])


def out_of_memory(e: RuntimeError) -> bool:
    """The device has no room (other failures of an allocation, a fault of an earlier kernel for one, are none of this)."""
    return "out of memory" in str(e)
