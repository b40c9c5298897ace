extern "C" const char* pb_abi() { return "1404724f9e58"; }
