"""ResNet-50 (bottleneck blocks [3, 4, 6, 3], 25.6M parameters) for the
image-classification data-parallel workload: many small gradient buckets, which
stresses the small-message (one-shot) path of the backend.  Plain PyTorch
layers; on channels-last activations BatchNorm, residual add and ReLU run as
one fused op (:func:`fairring_b200.ops.batch_norm_act`), and the pooling has
kernels of its own.
"""

from __future__ import annotations

import torch
import torch.nn as nn

from ..ops import batch_norm_act, max_pool, stem_conv
from ..ops._plain import native, plain_module


class Bottleneck(nn.Module):
    expansion = 4

    def __init__(self, inplanes: int, planes: int, stride: int = 1, downsample: nn.Module | None = None):
        super().__init__()
        self.conv1 = nn.Conv2d(inplanes, planes, 1, bias=False)
        self.bn1 = nn.BatchNorm2d(planes)
        self.conv2 = nn.Conv2d(planes, planes, 3, stride=stride, padding=1, bias=False)
        self.bn2 = nn.BatchNorm2d(planes)
        self.conv3 = nn.Conv2d(planes, planes * self.expansion, 1, bias=False)
        self.bn3 = nn.BatchNorm2d(planes * self.expansion)
        self.relu = nn.ReLU(inplace=True)
        self.downsample = downsample

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if not torch.jit.is_scripting():
            if native(x):
                return self.forward_pair(x, x)[0]
        identity = x if self.downsample is None else self.downsample(x)
        out = self.relu(self.bn1(self.conv1(x)))
        out = self.relu(self.bn2(self.conv2(out)))
        out = self.bn3(self.conv3(out))
        return self.relu(out + identity)

    def forward_pair(self, x: torch.Tensor, shortcut: torch.Tensor):
        """The block on an input that comes twice, for its convolutions and for its shortcut; so does
        the output, whose two gradients the backward then adds inside the BatchNorm."""
        identity, down = shortcut, self.downsample
        if down is not None and plain_module(down, nn.Sequential) and len(down) == 2:
            identity = batch_norm_act(down[1], down[0](shortcut))
        elif down is not None:
            identity = down(shortcut)
        out = batch_norm_act(self.bn1, self.conv1(x), relu=self.relu)
        out = batch_norm_act(self.bn2, self.conv2(out), relu=self.relu)
        return batch_norm_act(self.bn3, self.conv3(out), residual=identity, relu=self.relu, twice=True)


class ResNet50(nn.Module):
    def __init__(self, num_classes: int = 1000, layers=(3, 4, 6, 3), width: int = 64):
        super().__init__()
        self.inplanes = width
        self.conv1 = nn.Conv2d(3, width, 7, stride=2, padding=3, bias=False)
        self.bn1 = nn.BatchNorm2d(width)
        self.relu = nn.ReLU(inplace=True)
        self.maxpool = nn.MaxPool2d(3, stride=2, padding=1)
        self.layer1 = self._make_layer(width, layers[0])
        self.layer2 = self._make_layer(width * 2, layers[1], stride=2)
        self.layer3 = self._make_layer(width * 4, layers[2], stride=2)
        self.layer4 = self._make_layer(width * 8, layers[3], stride=2)
        self.avgpool = nn.AdaptiveAvgPool2d(1)
        self.fc = nn.Linear(width * 8 * Bottleneck.expansion, num_classes)
        for m in self.modules():
            if isinstance(m, nn.Conv2d):
                nn.init.kaiming_normal_(m.weight, mode="fan_out", nonlinearity="relu")
            elif isinstance(m, nn.BatchNorm2d):
                nn.init.ones_(m.weight)
                nn.init.zeros_(m.bias)

    def _make_layer(self, planes: int, blocks: int, stride: int = 1) -> nn.Sequential:
        downsample = None
        if stride != 1 or self.inplanes != planes * Bottleneck.expansion:
            downsample = nn.Sequential(
                nn.Conv2d(self.inplanes, planes * Bottleneck.expansion, 1, stride=stride, bias=False),
                nn.BatchNorm2d(planes * Bottleneck.expansion),
            )
        layers = [Bottleneck(self.inplanes, planes, stride, downsample)]
        self.inplanes = planes * Bottleneck.expansion
        layers += [Bottleneck(self.inplanes, planes) for _ in range(1, blocks)]
        return nn.Sequential(*layers)

    def num_parameters(self) -> int:
        return sum(p.numel() for p in self.parameters())

    def forward(self, images: torch.Tensor, labels: torch.Tensor | None = None):
        if not torch.jit.is_scripting():
            if native(images):
                return self._head(self._stages(images), labels)
        x = self.maxpool(self.relu(self.bn1(self.conv1(images))))
        x = self.layer4(self.layer3(self.layer2(self.layer1(x))))
        return self._head(x, labels)

    def _stages(self, images: torch.Tensor) -> torch.Tensor:
        """What stands in front of the pooling, on the ops of this package."""
        x = max_pool(self.maxpool, batch_norm_act(self.bn1, stem_conv(self.conv1, images), relu=self.relu))
        shortcut = x
        for stage in (self.layer1, self.layer2, self.layer3, self.layer4):
            if plain_module(stage, nn.Sequential) and all(plain_module(block, Bottleneck) for block in stage):
                for block in stage:
                    x, shortcut = block.forward_pair(x, shortcut)
            else:
                x = shortcut = stage(x)
        return x

    def _head(self, x: torch.Tensor, labels: torch.Tensor | None = None):
        logits = self.fc(torch.flatten(self.avgpool(x), 1))
        if labels is None:
            return logits
        return nn.functional.cross_entropy(logits.float(), labels)

    @staticmethod
    def tiny() -> "ResNet50":
        return ResNet50(num_classes=10, layers=(1, 1, 1, 1), width=8)
