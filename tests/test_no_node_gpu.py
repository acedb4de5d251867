"""Operators called without a gradient to carry skip the autograd node: same results, and what a node
refuses (tangents, functorch transforms) is still refused."""
import pytest
import torch
import torch.autograd.forward_ad as fwad

from tests.test_autograd_native_gpu import _traced_calls

pytestmark = pytest.mark.gpu


def test_same_results_with_and_without_a_node():
    for name, fn, args in _traced_calls():
        plain = [t.detach().clone() for t in args]
        with torch.no_grad():
            quiet = fn(*[t.clone() for t in plain])
        with torch.inference_mode():
            inferred = fn(*[t.clone() for t in plain])
        leaves = [t.clone().requires_grad_() for t in plain]
        loud = fn(*leaves)
        with torch.no_grad():
            muted = fn(*[t.clone().requires_grad_() for t in plain])
        assert loud.requires_grad, name
        for other in (fn(*plain), quiet, inferred, muted):
            assert not other.requires_grad and other.grad_fn is None, name
            torch.testing.assert_close(other.clone(), loud.detach(), msg=lambda m, n=name: f"{n}: {m}")


def test_tangents_and_transforms_are_still_refused():
    for name, fn, args in _traced_calls():
        plain = [t.detach().clone() for t in args]
        for grad_mode in (True, False):
            with fwad.dual_level(), torch.set_grad_enabled(grad_mode):
                dual = fwad.make_dual(plain[0], torch.ones_like(plain[0]))
                with pytest.raises(RuntimeError):
                    fn(dual, *plain[1:])
        with pytest.raises(RuntimeError), torch.no_grad():
            torch.func.vmap(lambda x: fn(x, *plain[1:]))(torch.stack([plain[0], plain[0]]))
