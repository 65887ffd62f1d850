"""Shapes by the kernel form that the library chooses for them: tests/test_host_dispatch.py asserts the choice without a GPU, the GPU
tests run the same shapes."""

# One layer (convolution of filter k, stride 1, padding k // 2, then ReLU and a pooling, so that its result stays NHWC) whose reduction
# is split: precision, (images, channels, h, w, output channels, k), CTAs of a cluster, channels of a tile. Every size of a cluster at
# every width it is chosen for; tiles of 128, 126, 121, 117, 98, 63, 9 and 1 pixels, whose rows divide unevenly among 3, 5, 6 and 7 owners
# (and among 8 when there are fewer than 8); last tiles of 32 to 96 channels.
SPLIT_LAYERS = [
    ("bf16", (50, 1024, 14, 9, 32, 1), 2, 64), ("bf16", (64, 768, 7, 7, 160, 1), 2, 128), ("bf16", (40, 768, 14, 9, 32, 1), 3, 64),
    ("bf16", (5, 768, 7, 7, 1600, 1), 3, 128), ("bf16", (28, 192, 13, 11, 160, 3), 3, 256), ("bf16", (24, 768, 14, 9, 32, 1), 4, 64),
    ("bf16", (3, 1536, 7, 7, 1600, 1), 4, 128), ("bf16", (20, 256, 13, 11, 160, 3), 4, 256), ("bf16", (24, 128, 8, 16, 32, 3), 5, 64),
    ("bf16", (5, 128, 7, 7, 1024, 3), 5, 128), ("bf16", (2, 768, 7, 7, 32, 1), 6, 64), ("bf16", (18, 128, 13, 11, 96, 3), 6, 128),
    ("bf16", (1, 192, 9, 7, 64, 3), 7, 64), ("bf16", (4, 192, 4, 6, 32, 3), 7, 64), ("bf16", (1, 192, 3, 3, 32, 3), 7, 64),
    ("bf16", (2, 1024, 7, 7, 32, 1), 8, 64), ("bf16", (1, 1024, 1, 1, 32, 1), 8, 64), ("bf16", (1, 320, 3, 3, 1600, 3), 8, 128),
    ("tf32", (50, 512, 14, 9, 32, 1), 2, 64), ("tf32", (64, 512, 7, 7, 160, 1), 2, 128), ("tf32", (64, 512, 7, 7, 320, 1), 2, 256),
    ("tf32", (40, 512, 14, 9, 32, 1), 3, 64), ("tf32", (5, 512, 7, 7, 1600, 1), 3, 128), ("tf32", (40, 512, 14, 9, 160, 1), 3, 256),
    ("tf32", (1, 512, 1, 1, 1600, 1), 4, 64), ("tf32", (3, 768, 7, 7, 1600, 1), 4, 128), ("tf32", (20, 128, 13, 11, 160, 3), 4, 256),
    ("tf32", (24, 768, 14, 9, 32, 1), 5, 64), ("tf32", (5, 768, 7, 7, 1024, 1), 5, 128), ("tf32", (40, 512, 7, 7, 32, 1), 6, 64),
    ("tf32", (11, 512, 14, 9, 224, 1), 6, 128), ("tf32", (2, 512, 7, 7, 32, 1), 8, 64), ("tf32", (28, 1536, 7, 7, 96, 1), 8, 128),
    ("tf32x3", (50, 512, 14, 9, 32, 1), 2, 64), ("tf32x3", (64, 768, 7, 7, 160, 1), 2, 128), ("tf32x3", (40, 512, 14, 9, 32, 1), 3, 64),
    ("tf32x3", (5, 512, 7, 7, 1600, 1), 3, 128), ("tf32x3", (3, 512, 7, 7, 1600, 1), 4, 128), ("tf32x3", (24, 768, 14, 9, 32, 1), 5, 64),
    ("tf32x3", (5, 768, 7, 7, 1024, 1), 5, 128), ("tf32x3", (40, 768, 7, 7, 96, 1), 6, 128), ("tf32x3", (1, 512, 1, 1, 32, 1), 8, 64),
    ("tf32x3", (28, 1024, 7, 7, 96, 1), 8, 128),
]


def split_layer(relay, case, to_constant, weight, bias):
    n, c, h, w, _, k = case
    x = relay.Var("input", (n, c, h, w))
    conv = relay.Call("nn_conv2d", [x, relay.Constant(to_constant(weight)), relay.Constant(to_constant(bias))],
                      relay.Conv2DAttrs((1, 1), (k // 2,) * 4, (1, 1), 1))
    pool = relay.MaxPool2DAttrs((1, 1), (1, 1, 1, 1), (1, 1), (3, 3), "NCHW", False)
    return relay.Function([x], relay.Call("nn_max_pool2d", [relay.Call("nn_relu", [conv])], pool))
