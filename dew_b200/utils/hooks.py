"""Whether anybody would notice that a module's call is made in another form, or not at all."""
from __future__ import annotations

from torch.nn.modules import module as _all


def moves_weights(hook):
    """Marks a forward hook that brings a module's weights and takes no notice of what the module is given."""
    hook.moves_weights = True
    return hook


def watched(module) -> bool:
    """Whether a forward hook of ``module``, of one inside it or of all modules may look at what they are given or return (those of ``moves_weights`` do not)."""
    if _all._global_forward_hooks or _all._global_forward_pre_hooks:
        return True
    return _watched(module)


def _watched(module) -> bool:
    own = module.__dict__
    for hooks in (own["_forward_hooks"], own["_forward_pre_hooks"]):
        for hook in hooks.values():
            if not getattr(hook, "moves_weights", False):
                return True
    for child in own["_modules"].values():
        if child is not None and _watched(child):
            return True
    return False


def nobody_watches_all() -> bool:
    """No hook that all modules have, in either direction."""
    return not (_all._global_forward_hooks or _all._global_forward_pre_hooks or _all._global_backward_hooks or _all._global_backward_pre_hooks)


def runs_alone_by_itself(module) -> bool:
    """``runs_alone`` but for the hooks of all modules."""
    own = module.__dict__
    return not ("forward" in own or own["_forward_hooks"] or own["_forward_pre_hooks"] or own["_backward_hooks"] or own["_backward_pre_hooks"])


def runs_alone(module) -> bool:
    """Whether calling ``module`` is running its class's ``forward`` and nothing else: no hook of its own or of all modules, in either direction, and no ``forward``
    set on the instance."""
    return runs_alone_by_itself(module) and nobody_watches_all()
