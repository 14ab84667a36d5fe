"""Softmax cross-entropy over logit rows as one library kernel (loss and gradient in the same launch): the loss the
reference's example networks train with (HUJI-Deep/simnets-tf README.md:108-111)."""
from .. import _lib
from .. import _torch_glue


def softmax_cross_entropy_with_grad(logits, labels, scale=1.0):
    """(loss, dlogits): loss = scale * sum_b (logsumexp(logits[b]) - logits[b, labels[b]]) as a 0-d tensor and its
    gradient with respect to the logits.  float32 CUDA logits [batch, classes], int64 CUDA labels [batch]."""
    return _lib.ops().xent_with_grad(logits, labels, float(scale))


def softmax_cross_entropy(logits, labels, scale=1.0):
    """Differentiable (w.r.t. the logits) form of softmax_cross_entropy_with_grad."""
    if _torch_glue.is_tracing():
        return _torch_glue.recorded(lambda l, k: _lib.ops().xent_apply(l, k, float(scale)), logits, labels)
    return _lib.ops().xent_apply(logits, labels, float(scale))
