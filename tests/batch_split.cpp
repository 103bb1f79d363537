// For each line "rest share sms count nodes [count nodes ...]" (uniform groups,
// largest first) prints how many of the fitting domains batch_split.h sends
// over every SM.
#include <cstdio>
#include <iostream>
#include <sstream>
#include <string>

#include "../lbm-c_b200/csrc/batch_split.h"

int main() {
  std::string line;
  while (std::getline(std::cin, line)) {
    std::istringstream in(line);
    long long rest, share, count, nodes;
    int sms;
    in >> rest >> share >> sms;
    std::vector<long long> fit;
    while (in >> count >> nodes) fit.insert(fit.end(), count, nodes);
    printf("%zu\n", lbmc::wide_of_fitting(fit, rest, share, sms));
  }
  return 0;
}
